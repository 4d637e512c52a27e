// serve_internal.h -- what the serving loops' kernels (serve.cu,
// serve_modes.cu) and their host share.
#pragma once

#include "rve_modes_kernel.cuh"

namespace sp {

constexpr int SERVE_NT = 512;
constexpr int SERVE_K = 7;  // eps and eps + delta e_i, i = 0..5 (component-major vectors need no padding)
constexpr int SERVE_NRHS = 7;
constexpr double FD_DELTA = 0.005;  // micro/inc/micro.h:29

struct ServeGeom {
  MeshGeo g;
  const int *cols;
  const int *nbr;
  float *vals;  // node-sliced ELL values [nn_pad*243] (assembled operator only)
  float *dinv;  // component-major [3][nn_pad]
  const uint8_t *etype;
  double *Ke;   // [2][576]
  double *D;    // [72]
  double *Bbar; // [144]
  double *warm;     // [SERVE_K][3][nn_pad] solutions of the previous request
  double *warm_eps; // [SERVE_K][6] its load-case strains
  double *gram;     // [6][6] b_i . b_j of the unit-strain right-hand sides b_i = -K u_bc(e_i)
  const int *color_elems;
  const uint8_t *slot;
  int color_off[9];
  // element-mode loop (serve_modes.cu)
  double mats[4], len[3];
  int on, cube;      // vectors on chip; equal element edges
  int wlen, pad;
  double *store;     // two stores of ([SERVE_NRHS][3][wlen] fluctuations, [SERVE_NRHS][6] strains)
  unsigned gen;      // published stores so far, the last one in store gen & 1
                     // (serve.cu's loop: twice the stores, odd while one is written)
  unsigned lock;     // 1: a request in flight writes a store
};

struct ServeReq {
  int geom, pad;
  double strain[6];
};

struct ServeRes {
  double stress[6];
  double tangent[36];
  sp_solve_info info;
  volatile long long done; // ticket + 1 once the result is valid
};

struct ServeCtl { // mapped host memory
  volatile long long tail;
  volatile int stop;
  int pad;
};

struct ServeDev { // device memory
  unsigned long long claim;
  volatile long long dtail;
  volatile int dstop;
  volatile int dispatcher_gone;
  int lost;  // 1: a worker gave up a ticket, whose load case stays unsolved
};

// A request in the element-mode loop: its load cases are tasks of their own
struct ServeJob {
  unsigned left;    // load cases still to finish
  unsigned stored;  // bit k: load case k is in the geometry's other store
  unsigned met;     // bit k: ... met the tolerance as predicted from store gen[k]
  unsigned solved;  // load cases kept for more than their prediction
  unsigned gen[SERVE_NRHS];
  unsigned writer;  // 1: this request holds the geometry's lock; 0: undecided
  int status, outer, inner;
  unsigned long long relres;  // bits of the largest one (non-negative or NaN)
  double stress[SERVE_NRHS][6];
};

struct ServeModes {
  ServeGeom *geoms;
  int ngeom, cap;
  const ServeReq *hreq;  // mapped ring
  ServeReq *dreq;        // device rings
  ServeJob *jobs;
  ServeRes *res;         // mapped ring
  const ServeCtl *ctl;
  ServeDev *dev;         // claim counts load cases
  ModesBufs buf;
  ModesLimits lim;
  int idle_limit, warm_last, dyn;
};

// The element-mode loop's kernels: threads and CTAs per SM.  A server takes
// the smallest class that holds every geometry's p and q in shared memory
// beside the class's other CTAs, so that small geometries have several load
// cases in flight per SM; the last class also serves the larger ones.
struct ServeClass {
  int threads, ctas;
  double match;  // CTAs that serve at least as much as a slot of the former loop
  void (*fn)(const ServeModes);
  // dynamic shared memory of a CTA (static data and the driver's share apart)
  int dyn() const {
    const int room = 228 * 1024 / ctas - 2048;
    return (room < 226 * 1024 ? room : 226 * 1024) / 16 * 16;
  }
};
constexpr int SERVE_CLASSES = 4;
extern const ServeClass kServeClasses[SERVE_CLASSES];

}  // namespace sp
