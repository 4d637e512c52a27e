// rve_plain.cu -- the plain GPU path: one RVE at a time, FP64 throughout,
// every step a grid-wide kernel.  This is the reference's micro solve
// (micro/src/homogenize.c:175-225, micro/src/assembly.c:33-137) moved to the
// GPU without batching or mixed precision: element operators, coloured
// scatter assembly into ELL, Dirichlet rows/columns, FP64 element residual,
// Jacobi-PCG (k_plain_pcg, or pcg.cuh's graph) and FP64 volume averages.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "pcg.cuh"
#include "sp_cuda.h"

namespace sp {

constexpr int KMAX = SP_MAX_RHS;

// element operators for the two materials: one block
__global__ void k_rve_ops(MeshGeo g, const double *D, double *Ke, double *Bbar) {
  __shared__ double dsh[192];
  double h[3] = {g.hx, g.hy, g.hz};
  elem_ops_stage1(threadIdx.x, blockDim.x, h, dsh);
  __syncthreads();
  elem_ops_stage2(threadIdx.x, blockDim.x, h, dsh, D, 2, Ke, Bbar);
}

template <typename T>
__global__ void k_zero_vals(T *vals, int ndof) {
  ell_zero<T>(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, vals, ndof);
}

template <typename T>
__global__ void k_scatter(MeshGeo g, const int *color_elems, int c0, int c1, const uint8_t *slot,
                          const uint8_t *etype, const double *Ke64, T *vals) {
  __shared__ T ke[2 * SP_KE];
  for (int x = threadIdx.x; x < 2 * SP_KE; x += blockDim.x) ke[x] = (T)Ke64[x];
  __syncthreads();
  scatter_colour<T>(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, g, color_elems,
                    c0, c1, slot, etype, ke, vals);
}

template <typename T>
__global__ void k_bc(MeshGeo g, const int *cols, T *vals, T *dinv) {
  bc_and_dinv<T>(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, g, cols, vals,
                 dinv);
}

template <int K>
__global__ void k_affine(MeshGeo g, const double *eps, int nrhs, double *u, bool inside) {
  affine_init<K>(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, g, eps, nrhs, u,
                 inside);
}

// Newton right-hand side b = -K u on interior dofs, 0 on boundary dofs
// (micro/src/assembly.c:33-82 then negative_res, micro/src/homogenize.c:
// 289-303), as the sum over the elements of the row's node of Ke_t[row][:] u_e
// (for linear elastic elements sum_gp B^T sigma(B u_e) w exactly);
// norms[k] = ||b_k||^2.  A thread per
// (row, load case), load cases fastest: a thread per row, with the K sums in
// registers, left 27,783 threads for n = 20 and waited on its loads (76 us,
// 6 load cases).
constexpr int RES_THREADS = 192;  // a multiple of K = 1, 6 and 8 load cases
template <int K>
__global__ void __launch_bounds__(RES_THREADS)
    k_residual(MeshGeo g, const uint8_t *__restrict__ etype, const double *Ke64,
               const double *__restrict__ u, double *b, double *norms, double *partial,
               unsigned *ticket) {
  __shared__ double ke[2 * SP_KE];
  __shared__ double red[33 * K];
  __shared__ double tot[K];
  __shared__ bool flag;
  for (int x = threadIdx.x; x < 2 * SP_KE; x += blockDim.x) ke[x] = Ke64[x];
  __syncthreads();
  const int q = threadIdx.x % K, nt = gridDim.x * (RES_THREADS / K);
  double nrm = 0.0;
  for (int row = (blockIdx.x * RES_THREADS + threadIdx.x) / K; row < g.ndof; row += nt) {
    const int node = row / 3, d = row % 3;
    const int i = node % g.nx, j = (node / g.nx) % g.ny, k = node / (g.nx * g.ny);
    double acc = 0.0;
    if (!is_bnode(g, node)) {
#pragma unroll 1
      for (int c = 0; c < 8; c++) {
        const int ox = c & 1, oy = (c >> 1) & 1, oz = c >> 2;
        const int ex = i - 1 + ox, ey = j - 1 + oy, ez = k - 1 + oz;
        // local index of this node in the element: corner (1-ox, 1-oy, 1-oz)
        const int cx = 1 - ox, cy = 1 - oy, cz = 1 - oz;
        const int la = cz * 4 + ((cy == 0) ? (cx ? 1 : 0) : (cx ? 2 : 3));
        const double *kr = ke + etype[ex + ey * g.nex + ez * g.nex * g.ney] * SP_KE +
                           (la * 3 + d) * SP_NC;
        const int n0 = ex + ey * g.nx + ez * g.nx * g.ny;
        double v[SP_NC];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
          for (int e = 0; e < 3; e++)
            v[a * 3 + e] = u[(size_t)(3 * (n0 + corner_x(a) + corner_y(a) * g.nx +
                                           corner_z(a) * g.nx * g.ny) + e) * K + q];
#pragma unroll
        for (int a = 0; a < SP_NC; a++) acc = fma(kr[a], v[a], acc);
      }
    }
    b[(size_t)row * K + q] = -acc;
    nrm += acc * acc;
  }
  double mine[K];
#pragma unroll
  for (int k = 0; k < K; k++) mine[k] = k == q ? nrm : 0.0;
  if (grid_sum<K>(mine, partial, ticket, red, tot, &flag) && threadIdx.x == 0)
    #pragma unroll
    for (int k = 0; k < K; k++) norms[k] = tot[k];
}

template <int K>
__global__ void k_add(int n, const double *x, double *u) {
  int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (int i = t; i < n * K; i += nt) u[i] += x[i];
}

// averages of load case q = blockIdx.y: out[0..5] strain, out[6..11] stress
template <int K>
__global__ void __launch_bounds__(256)
    k_average(MeshGeo g, const uint8_t *etype, const double *D, const double *Bbar,
              const double *u, double *out, double *partial, unsigned *ticket) {
  const int q = blockIdx.y;
  __shared__ double sD[72], sB[144];
  __shared__ double red[33 * 12];
  __shared__ double tot[12];
  __shared__ bool flag;
  for (int x = threadIdx.x; x < 72; x += blockDim.x) sD[x] = D[x];
  for (int x = threadIdx.x; x < 144; x += blockDim.x) sB[x] = Bbar[x];
  __syncthreads();
  double acc[12];
  #pragma unroll
  for (int v = 0; v < 12; v++) acc[v] = 0.0;
  average_elems<K>(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, g, etype, sD,
                   sB, u, q, acc);
  if (grid_sum<12>(acc, partial + (size_t)q * gridDim.x * 12, ticket + q, red, tot, &flag) &&
      threadIdx.x == 0)
    #pragma unroll
    for (int v = 0; v < 12; v++) out[q * 12 + v] = tot[v] / g.vol;
}

// u [ndof][K] -> out [nrhs][ndof]
template <int K>
__global__ void k_split(int n, int nrhs, const double *u, double *out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (int i = t; i < n * nrhs; i += nt) out[i] = u[(size_t)(i % n) * K + i / n];
}

struct PlainPcg {
  MeshGeo g;
  const double *vals, *dinv, *b;
  const int *cols;
  double *z, *x, *r, *q;  // z: D^-1 r, gathered by the other blocks
  double *u;              // += the solution
  PcgState *st;
  double *part_a, *part_b;
  int onchip;             // r, q, x in shared memory
};

// Jacobi-PCG of K load cases from x = 0 over the interior nodes in one
// cooperative launch, a block per SM with a contiguous range of nodes, a warp
// per node: the node's three rows have one column list, so a gathered value
// serves three rows, and the 3K sums are spread over the lanes, which own the
// node's vector entries.  Vectors that no other block reads stay in shared
// memory.  Only z = D^-1 r is gathered: p = z + beta p and q = A z + beta q
// (= A p) are local, so an iteration has two grid barriers, one after each
// reduction.  Every block folds the partial sums in the same order and takes
// the same exit.
//
// What bounds it: the latency of the two barriers and folds and of one gather
// (the matrix, 18 MB at n = 20, is re-read from L2).  Against three kernels
// an iteration in a graph, a warp per row: 53 -> 15 us an iteration at n = 20
// with 6 load cases.
constexpr int PLAIN_NT = 512;
template <int K>
__global__ void __launch_bounds__(PLAIN_NT, 1) k_plain_pcg(const __grid_constant__ PlainPcg P) {
  namespace cgr = cooperative_groups;
  cgr::grid_group grid = cgr::this_grid();
  constexpr int W = 3 * K, NW = PLAIN_NT / 32;
  extern __shared__ __align__(16) double plain_sm[];
  __shared__ double red[2][NW][W];
  __shared__ double tot[2 * K];
  const MeshGeo &g = P.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = gridDim.x, blk = blockIdx.x;
  const int mx = g.nx - 2, my = g.ny - 2, ni = mx * my * (g.nz - 2);
  const int c0 = (int)((long long)ni * blk / nb), m = (int)((long long)ni * (blk + 1) / nb) - c0;
  const int mmax = (ni + nb - 1) / nb;
  double *const p_s = plain_sm;
  double *const r_s = P.onchip ? p_s + (size_t)mmax * W : P.r;
  double *const q_s = P.onchip ? r_s + (size_t)mmax * W : P.q;
  double *const x_s = P.onchip ? q_s + (size_t)mmax * W : P.x;
  const int own = spread_index(W), k = own < 0 ? 0 : own % K, d = own < 0 ? 0 : own / K;
  auto node_of = [&](int li) {
    const int id = c0 + li;
    return 1 + id % mx + (1 + id / mx % my) * g.nx + (1 + id / (mx * my)) * g.nx * g.ny;
  };
  auto at = [&](int li, int node) { return (size_t)(P.onchip ? li : node) * W + own; };
  // per-block sums of NV values per load case -> part, grid barrier, totals
  auto sum = [&](double v0, double v1, int nv, double *part) {
    if (own >= 0) {
      red[0][warp][own] = v0;
      red[1][warp][own] = v1;
    }
    __syncthreads();
    for (int v = warp; v < nv * K; v += NW) {
      const double *e = &red[v / K][lane < NW ? lane : 0][v % K];
      double s = lane < NW ? e[0] + e[K] + e[2 * K] : 0.0;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) part[(size_t)v * nb + blk] = s;
    }
    grid.sync();
    for (int v = warp; v < nv * K; v += NW) {
      double s = 0.0;
      for (int i = lane; i < nb; i += 32) s += __ldcg(part + (size_t)v * nb + i);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) tot[v] = s;
    }
    __syncthreads();
  };
  const double rtol2 = P.st->rtol2;
  const int max_its = P.st->max_its, nrhs = P.st->nactive;
  // start: x = p = q = 0, r = b, z = D^-1 r (0 on the boundary); r.z, b.b
  const int t = blk * PLAIN_NT + threadIdx.x, nt = nb * PLAIN_NT;
  for (int node = t; node < g.nn; node += nt)
    if (is_bnode(g, node))
      for (int i = 0; i < W; i++) P.z[(size_t)node * W + i] = 0.0;
  double rz = 0.0, rr = 0.0;
  if (own >= 0)
    for (int li = warp; li < m; li += NW) {
      const int node = node_of(li);
      const size_t o = at(li, node);
      const double r = P.b[(size_t)node * W + own], z = P.dinv[node * 3 + d] * r;
      x_s[o] = q_s[o] = p_s[(size_t)li * W + own] = 0.0;
      r_s[o] = r;
      P.z[(size_t)node * W + own] = z;
      rz += r * z;
      rr += r * r;
    }
  sum(rz, rr, 2, P.part_b);
  // the scalars of this lane's load case, and how many are active in all
  double rho = tot[k], beta = 0.0;
  const double bb = tot[K + k];
  unsigned act = 0;
#pragma unroll
  for (int i = 0; i < K; i++) act |= (tot[K + i] > 0.0 && i < nrhs ? 1u : 0u) << i;
  __syncthreads();
  int its = 0;
  while (act && its < max_its) {
    double pq = 0.0;
    for (int li = warp; li < m; li += NW) {
      const int node = node_of(li);
      const double *vr = P.vals + (size_t)node * 3 * SP_WP;
      const int *cr = P.cols + (size_t)node * 3 * SP_WP;
      double a[W];
#pragma unroll
      for (int i = 0; i < W; i++) a[i] = 0.0;
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const int j = lane + 32 * s;
        if (j < SP_ELL_WIDTH) {
          const int c = __ldg(cr + j);
          const double v0 = __ldg(vr + j), v1 = __ldg(vr + SP_WP + j), v2 = __ldg(vr + 2 * SP_WP + j);
          double zv[K];
          load_k<double, K, false>(P.z + (size_t)(c < 0 ? 0 : c) * K, zv);
#pragma unroll
          for (int i = 0; i < K; i++) {
            a[i] = fma(v0, zv[i], a[i]);
            a[K + i] = fma(v1, zv[i], a[K + i]);
            a[2 * K + i] = fma(v2, zv[i], a[2 * K + i]);
          }
        }
      }
      const double az = spread_sum<W>(a);
      if (own >= 0) {
        const size_t o = at(li, node), op = (size_t)li * W + own;
        const double p = fma(beta, p_s[op], P.z[(size_t)node * W + own]);
        const double q = fma(beta, q_s[o], az);
        p_s[op] = p;
        q_s[o] = q;
        pq = fma(p, q, pq);
      }
    }
    sum(pq, 0.0, 1, P.part_a);
    const double alpha = (act >> k & 1) && tot[k] != 0.0 ? rho / tot[k] : 0.0;
    rz = rr = 0.0;
    if (own >= 0)
      for (int li = warp; li < m; li += NW) {
        const int node = node_of(li);
        const size_t o = at(li, node);
        x_s[o] = fma(alpha, p_s[(size_t)li * W + own], x_s[o]);
        const double r = fma(-alpha, q_s[o], r_s[o]), z = P.dinv[node * 3 + d] * r;
        r_s[o] = r;
        P.z[(size_t)node * W + own] = z;
        rz = fma(r, z, rz);
        rr = fma(r, r, rr);
      }
    sum(rz, rr, 2, P.part_b);
    its++;
    unsigned done = 0;
    if (tot[K + k] <= rtol2 * bb) done = 1u << k;
    done = __reduce_or_sync(0xffffffffu, own >= 0 ? done : 0u);
    act &= ~done;
    beta = (act >> k & 1) && rho != 0.0 ? tot[k] / rho : 0.0;
    if (act >> k & 1) rho = tot[k];
  }
  if (own >= 0)
    for (int li = warp; li < m; li += NW) {
      const int node = node_of(li);
      P.u[(size_t)node * W + own] += x_s[at(li, node)];
    }
  if (t == 0) {
    P.st->its = its;
    P.st->nactive = __popc(act);
  }
}

// Per-element strain and stress of load case q (micro/src/homogenize.c:
// 370-395, get_elem_properties): the Gauss-weighted means over the element,
// Bbar u_e / vol_elm and D_t Bbar u_e / vol_elm; u is [ndof][K].
template <int K>
__global__ void k_elem_fields(MeshGeo g, const uint8_t *__restrict__ etype, const double *D,
                              const double *Bbar, const double *__restrict__ u, int q,
                              double *strain_e, double *stress_e) {
  const double vol_elm = g.hx * g.hy * g.hz;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.nelm; e += gridDim.x * blockDim.x) {
    int nod[8];
    elem_nodes(g, e, nod);
    double eps[6] = {0, 0, 0, 0, 0, 0};
    for (int a = 0; a < 8; a++)
      for (int d = 0; d < 3; d++) {
        double uv = u[(size_t)(nod[a] * 3 + d) * K + q];
        for (int v = 0; v < 6; v++) eps[v] = fma(Bbar[v * 24 + a * 3 + d], uv, eps[v]);
      }
    const double *C = D + etype[e] * 36;
    for (int v = 0; v < 6; v++) {
      double sv = 0.0;
      for (int w = 0; w < 6; w++) sv = fma(C[v * 6 + w], eps[w], sv);
      strain_e[(size_t)e * 6 + v] = eps[v] / vol_elm;
      stress_e[(size_t)e * 6 + v] = sv / vol_elm;
    }
  }
}

static int blocks_for(Device *d, long long items, int per_block) {
  long long b = (items + per_block - 1) / per_block;
  long long cap = (long long)d->nsm * 4;
  if (b < 1) b = 1;
  return (int)(b < cap ? b : cap);
}

}  // namespace sp

using namespace sp;

struct sp_rve_s {
  sp_rve_desc desc;
  DevPlan *plan = nullptr;
  MeshGeo g;
  int nfiber = 0, dev = -1, last_launches = 0;
  uint8_t *etype_h = nullptr;
  uint8_t *d_etype = nullptr;
  double *d_D = nullptr, *d_Ke = nullptr, *d_Bbar = nullptr;
  double *d_vals = nullptr, *d_dinv = nullptr;
  double *d_u = nullptr, *d_b = nullptr, *d_x = nullptr, *d_r = nullptr, *d_p = nullptr,
         *d_q = nullptr;
  double *d_eps = nullptr, *d_out = nullptr, *d_partial = nullptr;
  PcgState *d_st = nullptr;
  unsigned *d_ticket = nullptr;
  PcgGraph<double, 1, 32> *pcg1 = nullptr;
  PcgGraph<double, 6, 32> *pcg6 = nullptr;
  PcgGraph<double, 8, 32> *pcg8 = nullptr;
  size_t bytes = 0;
  int last_k = 0, last_nrhs = 0;  // padded and actual load cases of the last solve
};

// The cooperative solve wants a block on as many SMs at once as it has work
// for, at most one each; a serving loop on the device may hold some of them
// for as long as requests come, so beside one the graph of small kernels runs.
// p has to fit the blocks' shared memory (n <= 54 with 8 load cases); larger
// RVEs stream the matrix from HBM either way.  Where the launch is refused (SMs
// held by another process's partition, say) the graph runs too.
template <int K>
static int plain_launch(sp_rve *r, Device *d, cudaStream_t s, bool *taken) {
  *taken = false;
  const MeshGeo &g = r->g;
  const long long ni = (long long)(g.nx - 2) * (g.ny - 2) * (g.nz - 2);
  if (ni < 1) return SP_OK;
  const int nb = (int)std::min<long long>(d->nsm, (ni + PLAIN_NT / 32 - 1) / (PLAIN_NT / 32));
  const size_t vec = (size_t)((ni + nb - 1) / nb) * 3 * K * sizeof(double), room = 200 * 1024;
  if (vec > room) return SP_OK;
  PlainPcg P = {g, r->d_vals, r->d_dinv, r->d_b, r->plan->cols, r->d_p, r->d_x, r->d_r, r->d_q,
                r->d_u, r->d_st, r->d_partial, r->d_partial + (size_t)d->nsm * 2 * K,
                4 * vec <= room};
  SP_CUDA_TRY(cudaFuncSetAttribute((const void *)k_plain_pcg<K>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
  void *args[] = {&P};
  bool refused = false;
  SP_TRY(d->gate.launch_alone(
      [&]() -> int {
        refused = cudaLaunchCooperativeKernel((const void *)k_plain_pcg<K>, dim3(nb), dim3(PLAIN_NT),
                                              args, P.onchip ? 4 * vec : vec, s) != cudaSuccess;
        if (!refused) SP_CUDA_TRY(cudaEventRecord(d->alone, s));
        return SP_OK;
      },
      taken));
  if (refused) {
    cudaGetLastError();  // (an error that outlasts the launch comes back from the graph)
    *taken = false;
  }
  return SP_OK;
}

static int rve_assemble(sp_rve *r, Device *d, cudaStream_t s) {
  MeshGeo &g = r->g;
  DevPlan *p = r->plan;
  k_rve_ops<<<1, SP_KE, 0, s>>>(g, r->d_D, r->d_Ke, r->d_Bbar);
  k_zero_vals<double><<<blocks_for(d, (long long)g.ndof * SP_WP / 2, 256), 256, 0, s>>>(r->d_vals,
                                                                                      g.ndof);
  for (int c = 0; c < 8; c++) {
    int c0 = p->color_off[c], c1 = p->color_off[c + 1];
    if (c1 == c0) continue;
    k_scatter<double><<<blocks_for(d, (long long)(c1 - c0) * SP_KE, 256), 256, 0, s>>>(
        g, p->color_elems, c0, c1, p->slot, r->d_etype, r->d_Ke, r->d_vals);
  }
  k_bc<double><<<blocks_for(d, g.ndof, 256), 256, 0, s>>>(g, p->cols, r->d_vals, r->d_dinv);
  SP_CUDA_TRY(cudaGetLastError());
  return SP_OK;
}

extern "C" int sp_rve_create(const sp_rve_desc *desc, sp_rve **out) {
  if (!desc || !out) return sp_set_error(SP_ERR_ARG, "sp_rve_create: null argument");
  for (int k = 0; k < 3; k++)
    if (desc->n[k] < 1 || desc->len[k] <= 0)
      return sp_set_error(SP_ERR_ARG, "sp_rve_create: bad mesh size or length");
  Device *d;
  SP_TRY(device(&d));
  sp_rve *r = new sp_rve_s();
  r->desc = *desc;
  r->dev = d->id;
  int rc = plan_acquire(desc->n, &r->plan);
  if (rc) {
    delete r;
    return rc;
  }
  r->g = make_geo(desc->n, desc->len);
  MeshGeo &g = r->g;
  r->etype_h = (uint8_t *)malloc(g.nelm);
  if (!r->etype_h) rc = sp_set_error(SP_ERR_NOMEM, "etype");
  if (!rc) rc = sp_classify_elements(desc, r->etype_h, &r->nfiber);
  size_t nv = (size_t)g.ndof * KMAX * sizeof(double);
  if (!rc) rc = dmalloc((void **)&r->d_etype, g.nelm, &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_D, 72 * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_Ke, 2 * SP_KE * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_Bbar, 144 * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_vals, (size_t)g.ndof * SP_WP * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_dinv, (size_t)g.ndof * sizeof(double), &r->bytes);
  double **vecs[6] = {&r->d_u, &r->d_b, &r->d_x, &r->d_r, &r->d_p, &r->d_q};
  for (int v = 0; v < 6 && !rc; v++) rc = dmalloc((void **)vecs[v], nv, &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_eps, KMAX * 6 * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_out, KMAX * 16 * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_partial, 4096 * 32 * sizeof(double), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_st, sizeof(PcgState), &r->bytes);
  if (!rc) rc = dmalloc((void **)&r->d_ticket, 64, &r->bytes);
  if (!rc) {
    double D[72];
    sp_iso_D(desc->E[0], desc->nu[0], D);
    sp_iso_D(desc->E[1], desc->nu[1], D + 36);
    cudaStream_t s = d->stream;
    if (cudaMemcpyAsync(r->d_etype, r->etype_h, g.nelm, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(r->d_D, D, sizeof(D), cudaMemcpyHostToDevice, s) ||
        cudaMemsetAsync(r->d_ticket, 0, 64, s))
      rc = sp_set_error(SP_ERR_CUDA, "sp_rve_create: upload failed");
    if (!rc) rc = rve_assemble(r, d, s);
    if (!rc && cudaStreamSynchronize(s))
      rc = sp_set_error(SP_ERR_CUDA, "sp_rve_create: assembly failed: %s",
                        cudaGetErrorString(cudaGetLastError()));
  }
  if (rc) {
    sp_rve_destroy(r);
    return rc;
  }
  *out = r;
  return SP_OK;
}

extern "C" int sp_rve_destroy(sp_rve *r) {
  if (!r) return SP_OK;
  delete r->pcg1;
  delete r->pcg6;
  delete r->pcg8;
  void *bufs[] = {r->d_etype, r->d_D, r->d_Ke, r->d_Bbar, r->d_vals, r->d_dinv, r->d_u,
                  r->d_b, r->d_x, r->d_r, r->d_p, r->d_q, r->d_eps, r->d_out, r->d_partial,
                  r->d_st, r->d_ticket};
  for (void *b : bufs) cudaFree(b);
  plan_release(r->plan);
  free(r->etype_h);
  delete r;
  return SP_OK;
}

extern "C" int sp_rve_sizes(const sp_rve *r, int *ndof, int *nelm, int *nfiber) {
  if (!r) return sp_set_error(SP_ERR_ARG, "null rve");
  if (ndof) *ndof = r->g.ndof;
  if (nelm) *nelm = r->g.nelm;
  if (nfiber) *nfiber = r->nfiber;
  return SP_OK;
}

extern "C" int sp_rve_get_ell(sp_rve *r, int *cols, double *vals) {
  if (!r) return sp_set_error(SP_ERR_ARG, "null rve");
  Device *d;
  SP_TRY(device(&d));
  size_t n = (size_t)r->g.ndof * SP_WP;
  int *hc = (int *)malloc(n * sizeof(int));
  double *hv = (double *)malloc(n * sizeof(double));
  int rc = (!hc || !hv) ? sp_set_error(SP_ERR_NOMEM, "staging") : SP_OK;
  if (!rc && (cudaMemcpy(hc, r->plan->cols, n * sizeof(int), cudaMemcpyDeviceToHost) ||
              cudaMemcpy(hv, r->d_vals, n * sizeof(double), cudaMemcpyDeviceToHost)))
    rc = sp_set_error(SP_ERR_CUDA, "sp_rve_get_ell: copy failed");
  if (!rc)
    for (int row = 0; row < r->g.ndof; row++) {
      if (cols) memcpy(cols + (size_t)row * SP_ELL_WIDTH, hc + (size_t)row * SP_WP, 81 * sizeof(int));
      if (vals)
        memcpy(vals + (size_t)row * SP_ELL_WIDTH, hv + (size_t)row * SP_WP, 81 * sizeof(double));
    }
  free(hc);
  free(hv);
  return rc;
}

extern "C" int sp_rve_get_ke(sp_rve *r, double *ke_matrix, double *ke_fiber) {
  if (!r) return sp_set_error(SP_ERR_ARG, "null rve");
  Device *d;
  SP_TRY(device(&d));
  double h[2 * SP_KE];
  SP_CUDA_TRY(cudaMemcpy(h, r->d_Ke, sizeof(h), cudaMemcpyDeviceToHost));
  if (ke_matrix) memcpy(ke_matrix, h, SP_KE * sizeof(double));
  if (ke_fiber) memcpy(ke_fiber, h + SP_KE, SP_KE * sizeof(double));
  return SP_OK;
}

template <int K>
static int rve_solve_k(sp_rve *r, Device *d, PcgGraph<double, K, 32> *&pcg, int nrhs,
                       const double *strains, double rtol, double *strain_ave, double *stress_ave,
                       double *u_out, sp_solve_info *info) {
  cudaStream_t s = d->stream;
  MeshGeo &g = r->g;
  int nb_res = blocks_for(d, (long long)g.ndof * K, RES_THREADS);
  int nb_vec = blocks_for(d, (long long)g.ndof * K, 256);
  int nb_row = blocks_for(d, g.ndof, PCG_THREADS / 32);
  int launches = 0;
  double eps[KMAX * 6] = {0};
  memcpy(eps, strains, (size_t)nrhs * 6 * sizeof(double));
  SP_CUDA_TRY(cudaMemcpyAsync(r->d_eps, eps, sizeof(eps), cudaMemcpyHostToDevice, s));
  k_affine<K><<<nb_vec, 256, 0, s>>>(g, r->d_eps, nrhs, r->d_u, false);
  launches++;
  double r0[KMAX] = {0}, rn[KMAX] = {0};
  int outer = 0, inner = 0, max_outer = 6;
  bool started = false;
  // Newton / refinement: b = -K u, solve A x = b, u += x  (micro/src/homogenize.c:184-215).
  // The first residual, of the boundary values alone, is the right-hand side
  // the stopping rule is relative to; the iteration then starts from the
  // homogeneous affine field eps . x inside (the exact solution for a
  // homogeneous RVE), which leaves the error near the material interfaces.
  for (;;) {
    double nrm[KMAX];
    k_residual<K><<<nb_res, RES_THREADS, 0, s>>>(g, r->d_etype, r->d_Ke, r->d_u, r->d_b, r->d_out + 8 * 12,
                                         r->d_partial, r->d_ticket);
    launches++;
    SP_CUDA_TRY(cudaMemcpyAsync(nrm, r->d_out + 8 * 12, K * sizeof(double), cudaMemcpyDeviceToHost, s));
    SP_CUDA_TRY(cudaStreamSynchronize(s));
    if (!started) {
      for (int k = 0; k < nrhs; k++) r0[k] = sqrt(nrm[k]);
      k_affine<K><<<nb_vec, 256, 0, s>>>(g, r->d_eps, nrhs, r->d_u, true);
      launches++;
      started = true;
      continue;
    }
    bool done = true;
    for (int k = 0; k < nrhs; k++) {
      rn[k] = sqrt(nrm[k]);
      if (r0[k] > 0 && rn[k] > rtol * r0[k]) done = false;
    }
    if (done || outer >= max_outer) break;
    PcgState st0 = {};
    st0.nactive = nrhs;
    st0.rtol2 = (0.5 * rtol) * (0.5 * rtol);
    st0.max_its = 20000;
    SP_CUDA_TRY(cudaMemcpyAsync(r->d_st, &st0, sizeof(st0), cudaMemcpyHostToDevice, s));
    int fixed = 0;
    bool coop;
    SP_TRY(plain_launch<K>(r, d, s, &coop));
    if (!coop) {
      if (!pcg) {
        pcg = new PcgGraph<double, K, 32>();
        SP_TRY(pcg->build(s, nb_row, g.ndof, SP_WP, r->d_vals, r->plan->cols, r->d_dinv, r->d_b,
                          r->d_x, r->d_r, r->d_p, r->d_q, 1, r->d_st, r->d_partial, r->d_ticket));
      }
      SP_TRY(pcg->run(s, &fixed));
      k_add<K><<<nb_vec, 256, 0, s>>>(g.ndof, r->d_x, r->d_u);
    }
    PcgState st;
    SP_CUDA_TRY(cudaMemcpyAsync(&st, r->d_st, sizeof(st), cudaMemcpyDeviceToHost, s));
    SP_CUDA_TRY(cudaStreamSynchronize(s));
    launches += coop ? 1 : fixed + 3 * st.its + 1;
    inner += st.its;
    outer++;
  }
  k_average<K><<<dim3(blocks_for(d, g.nelm, 256), nrhs), 256, 0, s>>>(
      g, r->d_etype, r->d_D, r->d_Bbar, r->d_u, r->d_out, r->d_partial, r->d_ticket);
  launches++;
  double out[KMAX * 12];
  SP_CUDA_TRY(cudaMemcpyAsync(out, r->d_out, sizeof(out), cudaMemcpyDeviceToHost, s));
  if (u_out) {
    // u is [ndof][K]; the caller wants [nrhs][ndof]
    k_split<K><<<nb_vec, 256, 0, s>>>(g.ndof, nrhs, r->d_u, r->d_x);
    launches++;
    SP_CUDA_TRY(cudaMemcpyAsync(u_out, r->d_x, (size_t)g.ndof * nrhs * sizeof(double),
                                cudaMemcpyDeviceToHost, s));
  }
  SP_CUDA_TRY(cudaStreamSynchronize(s));
  double worst = 0.0;
  for (int k = 0; k < nrhs; k++) {
    if (strain_ave) memcpy(strain_ave + 6 * k, out + 12 * k, 6 * sizeof(double));
    if (stress_ave) memcpy(stress_ave + 6 * k, out + 12 * k + 6, 6 * sizeof(double));
    double rel = r0[k] > 0 ? rn[k] / r0[k] : 0.0;
    if (rel > worst) worst = rel;
  }
  r->last_launches = launches;
  r->last_k = K;
  r->last_nrhs = nrhs;
  int status = (worst <= rtol) ? SP_OK : SP_ERR_NOCONV;
  if (info) {
    info->status = status;
    info->outer_its = outer;
    info->inner_its = inner;
    info->pad = launches;
    info->relres = worst;
  }
  return status ? sp_set_error(status, "plain solve stopped at relres %.3e", worst) : SP_OK;
}

extern "C" int sp_rve_homogenize(sp_rve *r, int nrhs, const double *strains, double rtol,
                                 double *strain_ave, double *stress_ave, double *u_out,
                                 sp_solve_info *info) {
  if (!r || !strains || nrhs < 1 || nrhs > KMAX || !(rtol > 0))
    return sp_set_error(SP_ERR_ARG, "sp_rve_homogenize: bad argument");
  Device *d;
  SP_TRY(device(&d));
  if (nrhs == 1)
    return rve_solve_k<1>(r, d, r->pcg1, nrhs, strains, rtol, strain_ave, stress_ave, u_out, info);
  if (nrhs <= 6)
    return rve_solve_k<6>(r, d, r->pcg6, nrhs, strains, rtol, strain_ave, stress_ave, u_out, info);
  return rve_solve_k<8>(r, d, r->pcg8, nrhs, strains, rtol, strain_ave, stress_ave, u_out, info);
}

extern "C" int sp_rve_tangent(sp_rve *r, double rtol, double *C, sp_solve_info *info) {
  if (!r || !C) return sp_set_error(SP_ERR_ARG, "sp_rve_tangent: null argument");
  double eps[36] = {0}, st[36];
  for (int j = 0; j < 6; j++) eps[j * 6 + j] = 1.0;
  int rc = sp_rve_homogenize(r, 6, eps, rtol, nullptr, st, nullptr, info);
  for (int i = 0; i < 6; i++)
    for (int j = 0; j < 6; j++) C[i * 6 + j] = st[j * 6 + i];
  return rc;
}

extern "C" int sp_rve_fields(sp_rve *r, int q, double *strain_e, double *stress_e, double *u,
                             double *residual) {
  if (!r) return sp_set_error(SP_ERR_ARG, "sp_rve_fields: null rve");
  if (r->last_nrhs < 1) return sp_set_error(SP_ERR_STATE, "sp_rve_fields: no solve yet");
  if (q < 0 || q >= r->last_nrhs)
    return sp_set_error(SP_ERR_RANGE, "sp_rve_fields: load case %d of %d", q, r->last_nrhs);
  Device *d;
  SP_TRY(device(&d));
  cudaStream_t s = d->stream;
  const MeshGeo &g = r->g;
  const size_t ne = (size_t)g.nelm * 6;
  double *dev = nullptr;
  SP_TRY(dmalloc((void **)&dev, 2 * ne * sizeof(double), nullptr));
  int nb = blocks_for(d, g.nelm, 256);
  switch (r->last_k) {
    case 1: k_elem_fields<1><<<nb, 256, 0, s>>>(g, r->d_etype, r->d_D, r->d_Bbar, r->d_u, q, dev, dev + ne); break;
    case 6: k_elem_fields<6><<<nb, 256, 0, s>>>(g, r->d_etype, r->d_D, r->d_Bbar, r->d_u, q, dev, dev + ne); break;
    default: k_elem_fields<8><<<nb, 256, 0, s>>>(g, r->d_etype, r->d_D, r->d_Bbar, r->d_u, q, dev, dev + ne); break;
  }
  cudaError_t e = cudaGetLastError();
  if (!e && strain_e) e = cudaMemcpyAsync(strain_e, dev, ne * sizeof(double), cudaMemcpyDeviceToHost, s);
  if (!e && stress_e) e = cudaMemcpyAsync(stress_e, dev + ne, ne * sizeof(double), cudaMemcpyDeviceToHost, s);
  // u and the last residual are [ndof][K]: one strided column each
  if (!e && u)
    e = cudaMemcpy2DAsync(u, sizeof(double), r->d_u + q, r->last_k * sizeof(double), sizeof(double),
                          g.ndof, cudaMemcpyDeviceToHost, s);
  if (!e && residual)
    e = cudaMemcpy2DAsync(residual, sizeof(double), r->d_b + q, r->last_k * sizeof(double),
                          sizeof(double), g.ndof, cudaMemcpyDeviceToHost, s);
  if (!e) e = cudaStreamSynchronize(s);
  cudaFree(dev);
  if (e) return sp_set_error(SP_ERR_CUDA, "sp_rve_fields: %s", cudaGetErrorString(e));
  return SP_OK;
}

extern "C" int sp_rve_write_vtu(sp_rve *r, int q, const char *base) {
  if (!r || !base) return sp_set_error(SP_ERR_ARG, "sp_rve_write_vtu: null argument");
  const MeshGeo &g = r->g;
  std::vector<double> se((size_t)g.nelm * 6), st((size_t)g.nelm * 6), u(g.ndof), res(g.ndof);
  SP_TRY(sp_rve_fields(r, q, se.data(), st.data(), u.data(), res.data()));
  return sp_vtu_write(base, r->desc.n, r->desc.len, u.data(), res.data(), r->etype_h, se.data(),
                      st.data());
}
