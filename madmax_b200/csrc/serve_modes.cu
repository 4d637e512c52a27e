// serve_modes.cu -- the element-mode request loop: serve.cu's loop with a CTA
// per load case of a request instead of one per request.
//
// A request's 7 load cases (eps and eps + delta e_i, micro/src/
// homogenize.c:59-94) are tasks of their own, claimed in order by the worker
// CTAs; the last one to finish forms the tangent, writes the result and
// raises the done flag.  A task runs the solve of rve_modes_kernel.cuh, whose
// vectors stay on chip where they fit, started from the geometry's store of
// the last solved request's fluctuations.
//
// Stores.  A geometry has two: the published one and the one being written.
// A request takes the geometry's lock when its first load case is claimed;
// without it, it stores nothing.  Its solutions go to the other store and are
// published (gen + 1) once all 7 are there.  Where some load cases were solved
// and others met the tolerance on their prediction, the request's last task
// adds the predictions, formed again from the published store, which stands
// as long as the lock is held; a request that met all of its predictions
// publishes nothing.  A task that read the published
// store while a later request's solutions replaced it (gen has moved on)
// starts cold instead, so no task starts from a mixture of two requests.
// Nothing waits: a lock that is taken is passed by.
//
// What bounds it: a task's set-up and its two residual passes where the
// prediction holds, the march of the corrections where it does not (the rate
// of k_modes).  Several CTAs per SM hide the set-up's loads (the classes of
// serve_internal.h); a task's time is a seventh of a request's, so a burst
// ends without a long last request.
#include "serve_internal.h"
#include "serve_ticket.h"

namespace sp {

struct ServeShared {
  long long req;  // ticket, -1: leave
  int geom, k, gen, stored;
  int last;       // the request's last task: 1, and 2 to publish its solutions
  unsigned fill;  // ... after adding the predictions of these load cases
  double eps[SERVE_NRHS][6];
  double c[6];  // prediction coefficients
  double rn0;
};

// first-order prediction of a load case of strain e from the solutions w_k of
// a store's strains: w = w_0 + sum_j c_j (w_j+1 - w_0)
__device__ __forceinline__ const double *serve_store(const ServeGeom &G, unsigned gen) {
  return G.store + (size_t)(gen & 1u) * SERVE_NRHS * (3 * G.wlen + 6);
}
__device__ __noinline__ void serve_coefs(const ServeGeom &G, unsigned gen, const double *e, double *c) {
  const double *se = serve_store(G, gen) + (size_t)SERVE_NRHS * 3 * G.wlen;
  for (int j = 0; j < 6; j++) {
    const double b = __ldcg(se + j), d = __ldcg(se + (j + 1) * 6 + j) - b;
    c[j] = d != 0.0 ? (e[j] - b) / d : 0.0;
  }
}
__device__ __forceinline__ double serve_predict(const double *st, int n, const double (&c)[6], int i) {
  const double w0 = __ldcg(st + i);
  double v[6];
#pragma unroll
  for (int j = 0; j < 6; j++) v[j] = __ldcg(st + (size_t)(j + 1) * n + i);
  double s = w0;
#pragma unroll
  for (int j = 0; j < 6; j++) s = fma(c[j], v[j] - w0, s);
  return s;
}

// Claim the next load case; one thread.  When work is published a CTA takes
// the next ticket and keeps it (serve_ticket.h): another may have taken the
// last published one in between, so it waits for its own to be published.
// (With a compare-and-swap on the counter the CTAs of the die far from it lost
// every race: half of them served nothing, and three passes over 6,912 points
// with n = 12 RVEs took 38.4 ms instead of 17.6 ms.)
__device__ __noinline__ void serve_claim(const ServeModes &P, ServeShared &S) {
  ServeDev *D = P.dev;
  ServeWait wait;
  long long task;
  for (;;) {
    const bool gone = D->dstop || D->dispatcher_gone;
    __threadfence();
    task = serve_poll(
        wait, gone, D->dtail * SERVE_NRHS, P.idle_limit,
        [&] { return (long long)*(volatile unsigned long long *)&D->claim; },
        [&] { return (long long)atomicAdd(&D->claim, 1ull); });
    if (task != SERVE_WAIT) break;
    __nanosleep(500);
  }
  if (task == SERVE_LOST) atomicExch(&D->lost, 1);
  __threadfence();
  S.req = task < 0 ? -1 : task / SERVE_NRHS;
  if (task < 0) return;
  S.k = (int)(task % SERVE_NRHS);
  const ServeReq *rq = P.dreq + S.req % P.cap;
  const int gid = __ldcg(&rq->geom);
  S.geom = gid;
  double e0[6];
  for (int j = 0; j < 6; j++) e0[j] = __ldcg(&rq->strain[j]);
  for (int c = 0; c < SERVE_NRHS; c++)
    for (int j = 0; j < 6; j++) S.eps[c][j] = e0[j] + (c == j + 1 ? FD_DELTA : 0.0);
  if (gid < 0 || gid >= P.ngeom) return;
  ServeGeom &G = P.geoms[gid];
  if (S.k == 0)
    atomicExch(&P.jobs[S.req % P.cap].writer, atomicCAS(&G.lock, 0u, 1u) == 0u ? 1u : 2u);
  S.gen = (int)atomicAdd(&G.gen, 0u);
  __threadfence();
  const double *e = S.eps[S.k];
  double s = 0.0;
  for (int a = 0; a < 6; a++)
    for (int b = 0; b < 6; b++) s += e[a] * __ldg(G.gram + a * 6 + b) * e[b];
  S.rn0 = s <= 0.0 ? 0.0 : sqrt(s);  // (a NaN stays one)
  if (S.gen) serve_coefs(G, S.gen, e, S.c);
}

// whether the request's last task publishes its solutions, and the load cases
// whose predictions belong to them; one thread
__device__ __noinline__ void serve_finish(ServeJob &J, ServeGeom &G, ServeShared &S) {
  if (atomicAdd(&J.writer, 0u) != 1u || atomicAdd(&J.solved, 0u) == 0u) return;
  const unsigned gen = atomicAdd(&G.gen, 0u), stored = atomicAdd(&J.stored, 0u),
                 met = atomicAdd(&J.met, 0u) & ~stored;
  for (int k = 0; k < SERVE_NRHS; k++)
    if ((met >> k & 1u) && *(volatile unsigned *)(J.gen + k) == gen) S.fill |= 1u << k;
  if ((stored | S.fill) == (1u << SERVE_NRHS) - 1)
    S.last = 2;
  else
    S.fill = 0;
}

// the start iterate: the fluctuation of the last solution of this load case
// (last), or predicted to first order from the 7 of the last solved request,
// or (cold) none.  modes_setup left w = -eps.x inside, which stays for a load
// case without a right-hand side.
__device__ __noinline__ void serve_start(const ServeGeom &G, ServeShared &S, bool last, double *w) {
  if (!(S.rn0 > 0.0)) return;
  const int n = 3 * G.wlen, t = threadIdx.x;
  const double *st = serve_store(G, S.gen);
  if (S.gen && last) {
    for (int i = t; i < n; i += blockDim.x) w[i] = __ldcg(st + (size_t)S.k * n + i);
  } else if (S.gen) {
    double c[6];
#pragma unroll
    for (int j = 0; j < 6; j++) c[j] = S.c[j];
    for (int i = t; i < n; i += blockDim.x) w[i] = serve_predict(st, n, c, i);
  }
  __syncthreads();
  if (S.gen) {
    if (t == 0) {
      __threadfence();
      if ((int)atomicAdd(const_cast<unsigned *>(&G.gen), 0u) != S.gen) S.gen = 0;
    }
    __syncthreads();
  }
  if (!S.gen)
    for (int i = t; i < n; i += blockDim.x) w[i] = 0.0;
  __syncthreads();
}

// the predictions of the load cases S.fill into the store being written
__device__ __noinline__ void serve_fill(ServeGeom &G, const ServeShared &S) {
  const int n = 3 * G.wlen, t = threadIdx.x;
  const unsigned gen = atomicAdd(&G.gen, 0u);
  const double *from = serve_store(G, gen);
  double *to = const_cast<double *>(serve_store(G, gen + 1));
#pragma unroll 1
  for (int k = 0; k < SERVE_NRHS; k++) {
    if (!(S.fill >> k & 1u)) continue;
    double c[6];
    serve_coefs(G, gen, S.eps[k], c);
    for (int i = t; i < n; i += blockDim.x)
      __stcg(to + (size_t)k * n + i, serve_predict(from, n, c, i));
    if (t < 6) __stcg(to + (size_t)SERVE_NRHS * n + k * 6 + t, S.eps[k][t]);
  }
  __threadfence();
  __syncthreads();
}

// one load case; thread 0 writes its stress average.  Returns its relative
// residual, NaN for a strain without a finite right-hand side (which is left
// without a step).
template <bool CUBE, int ON>
__device__ __noinline__ double serve_case(const ServeModes &P, const ServeGeom &G, ServeShared &S,
                                          double *stress) {
  ModesShared &sh = msh();
  if (threadIdx.x == 0) {
    const ModesGeo M(G.g.nex, G.g.ney, G.g.nez, false, false, ON);
    modes_sizes(M, sh);
  }
  __syncthreads();
  int ph = 0;
  {
    const ModesSpace<F2, ON> ws(P.buf);
    modes_setup<false, false>(G.len, G.mats, G.etype, S.eps[S.k], ws.w, ws.r);
    serve_start(G, S, P.warm_last, ws.w);
  }
  const double relres = modes_refine<F2, CUBE, ON, false>(P.buf, P.lim, S.rn0, ph);
  {
    const ModesSpace<F2, ON> ws(P.buf);
    march_average<false>(ws.w, ph);
  }
  if (threadIdx.x == 0) modes_output(sh.red, stress, nullptr);
  return isfinite(S.rn0) ? relres : nan("");
}

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_serve_modes(const __grid_constant__ ServeModes P) {
  __shared__ ServeShared S;
  const int t = threadIdx.x;
  ServeDev *D = P.dev;
  if (blockIdx.x == 0) {
    // dispatcher: forward host requests into the device ring
    if (t >= 32) return;
    long long seen = D->dtail;
    int idle = 0;
    for (;;) {
      long long ht = 0;
      int hstop = 0;
      if (t == 0) {
        ht = P.ctl->tail;
        hstop = P.ctl->stop;
      }
      ht = __shfl_sync(0xffffffffu, ht, 0);
      hstop = __shfl_sync(0xffffffffu, hstop, 0);
      __threadfence_system();
      if (ht > seen) {
        for (long long i = seen + t; i < ht; i += 32) {
          const volatile ServeReq *src = P.hreq + (i % P.cap);
          ServeReq *dst = P.dreq + (i % P.cap);
          dst->geom = src->geom;
          for (int k = 0; k < 6; k++) dst->strain[k] = src->strain[k];
          ServeJob &J = P.jobs[i % P.cap];
          J.left = SERVE_NRHS;
          J.stored = J.met = J.solved = J.writer = 0;
          J.status = J.outer = J.inner = 0;
          J.relres = 0;
        }
        __threadfence();
        __syncwarp();
        if (t == 0) D->dtail = ht;
        seen = ht;
        idle = 0;
      } else if (hstop) {
        __threadfence();  // the last publication first
        if (t == 0) D->dstop = 1;
        break;
      } else if (++idle > P.idle_limit) {
        break;
      }
      __nanosleep(1000);
    }
    if (t == 0) {
      __threadfence();
      D->dispatcher_gone = 1;
    }
    return;
  }
  if (dynamic_smem_bytes() < (unsigned)P.dyn) return;  // (the host's waits are bounded)
  for (;;) {
    if (t == 0) serve_claim(P, S);
    __syncthreads();
    if (S.req < 0) break;
    ServeJob &J = P.jobs[S.req % P.cap];
    const bool known = S.geom >= 0 && S.geom < P.ngeom;
    double relres = 0.0;
    if (known) {
      ServeGeom &G = P.geoms[S.geom];
      double *const stress = J.stress[S.k];
      switch (2 * G.on + (G.cube ? 1 : 0)) {
        case 5: relres = serve_case<true, 2>(P, G, S, stress); break;
        case 4: relres = serve_case<false, 2>(P, G, S, stress); break;
        default:
          if constexpr (MINB == 1) {  // only the last class serves these
            switch (2 * G.on + (G.cube ? 1 : 0)) {
              case 3: relres = serve_case<true, 1>(P, G, S, stress); break;
              case 2: relres = serve_case<false, 1>(P, G, S, stress); break;
              case 1: relres = serve_case<true, 0>(P, G, S, stress); break;
              default: relres = serve_case<false, 0>(P, G, S, stress); break;
            }
          }
      }
      // keep this load case's solution for the geometry's next requests when
      // it was solved (it then meets the refined tolerance); one accepted on
      // its prediction leaves the solved state in place, so predictions do
      // not drift from it.  One that is no nearer than a cold start (a residual
      // of 1) or not a number is no start for the next.
      if (t == 0) {
        const bool solved = msh().outer > 0 || S.gen == 0 || P.warm_last;
        S.stored = (solved || !(S.rn0 > 0.0)) && relres < 1.0 && atomicAdd(&J.writer, 0u) == 1u;
        if (S.stored && solved) atomicAdd(&J.solved, 1u);
        if (!solved && S.rn0 > 0.0 && relres <= P.lim.rtol) {
          J.gen[S.k] = (unsigned)S.gen;  // (fenced before left counts down)
          atomicOr(&J.met, 1u << S.k);
        }
      }
      if (t == 0) __threadfence();
      __syncthreads();
      if (S.stored) {
        const int n = 3 * G.wlen;
        double *st = const_cast<double *>(serve_store(G, atomicAdd(&G.gen, 0u) + 1));
        const double *w = P.buf.ws_w + (size_t)blockIdx.x * P.buf.w_stride;
        for (int i = t; i < n; i += blockDim.x) __stcg(st + (size_t)S.k * n + i, w[i]);
        if (t < 6) __stcg(st + (size_t)SERVE_NRHS * n + S.k * 6 + t, S.eps[S.k][t]);
      }
      __threadfence();
      __syncthreads();
    }
    if (t == 0) {
      if (known) {
        const int status = relres <= P.lim.rtol ? SP_OK : SP_ERR_NOCONV;
        atomicMax(&J.status, status);
        atomicMax(&J.outer, msh().outer);
        atomicMax(&J.inner, msh().inner);
        // (bits of a non-negative number grow with it, and NaN's are above all)
        atomicMax(&J.relres, (unsigned long long)__double_as_longlong(relres >= 0.0 ? relres : nan("")));
        if (S.stored) atomicOr(&J.stored, 1u << S.k);
      } else {
        atomicMax(&J.status, SP_ERR_RANGE);
      }
      __threadfence();
      S.last = atomicSub(&J.left, 1u) == 1u;
      S.fill = 0;
      if (S.last && known) {
        __threadfence();
        serve_finish(J, P.geoms[S.geom], S);
      }
    }
    __syncthreads();
    if (S.last) {
      if (S.fill) serve_fill(P.geoms[S.geom], S);
      if (t == 0) {
        __threadfence();
        ServeRes *out = P.res + (S.req % P.cap);
        if (known) {
          ServeGeom &G = P.geoms[S.geom];
          const volatile double(*st)[6] = J.stress;
          for (int v = 0; v < 6; v++) out->stress[v] = st[0][v];
          // c_tangent[j*6 + i] = (stress(eps + d e_i)_j - stress(eps)_j) / (d e_i)
          // (micro/src/homogenize.c:79-80)
          for (int i = 0; i < 6; i++)
            for (int j = 0; j < 6; j++)
              out->tangent[j * 6 + i] = (st[i + 1][j] - st[0][j]) / (S.eps[i + 1][i] - S.eps[0][i]);
          if (atomicAdd(&J.writer, 0u) == 1u) {
            if (S.last == 2) atomicAdd(&G.gen, 1u);
            __threadfence();
            atomicExch(&G.lock, 0u);
          }
        }
        sp_solve_info in = {};
        in.status = atomicAdd(&J.status, 0);
        in.outer_its = atomicAdd(&J.outer, 0);
        in.inner_its = atomicAdd(&J.inner, 0);
        in.relres = __longlong_as_double((long long)atomicAdd(&J.relres, 0ull));
        out->info = in;
        __threadfence_system();
        out->done = S.req + 1;
      }
    }
    __syncthreads();
  }
}

// 128 registers a thread at every class; the shared memory of a CTA is the
// SM's over its CTAs, so a class ends where p and q of a geometry no longer fit.
// Requests a second that a CTA serves, few of them at once, solved and
// predicted, against a slot of the former loop (512 threads): n = 6 1,092 and
// 5,470 against 2,037 and 7,380; n = 12 285 and 3,430 against 312 and 3,020;
// n = 16 167 and 2,670 against 111 and 1,650; n = 20 80 and 1,910 against 48 and
// 925; n = 28 11.4 and 663 against 10.5 and 362.
const ServeClass kServeClasses[SERVE_CLASSES] = {{64, 8, 2.0, k_serve_modes<64, 8>},
                                                 {160, 3, 1.1, k_serve_modes<160, 3>},
                                                 {256, 2, 1.0, k_serve_modes<256, 2>},
                                                 {512, 1, 1.0, k_serve_modes<512, 1>}};

}  // namespace sp
