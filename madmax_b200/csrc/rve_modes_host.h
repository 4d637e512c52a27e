// rve_modes_host.h -- host side of the element-mode batch kernel
// (rve_modes_kernel.cuh): which RVEs it takes, in which launches.
#pragma once

#include <vector>

#include "rve_modes_kernel.cuh"

namespace sp {

// one launch: RVEs of one kernel class, its persistent grid and work spaces
struct ModesBucket {
  ModesFn fn = nullptr;
  int threads = 0, grid = 0, smem = 0, nrve = 0;
  int *d_order = nullptr;
  double *ws_w = nullptr;
  void *ws_v = nullptr, *ws_e = nullptr;
  size_t w_stride = 0, v_stride = 0, e_stride = 0, v_cta = 0, bytes = 0;
};

// The launches of a batch: every bucket but the first on a side stream of its
// own, forked from the caller's stream and joined to it (which a stream
// capture records as parallel branches), so that one bucket's last CTAs
// overlap with the others.
struct ModesPlan {
  std::vector<ModesBucket> buckets;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> joined;
  cudaEvent_t forked = nullptr;
};

// What the launches of one batch share
struct ModesCommon {
  const BatchPlan *plans;
  const BatchRve *rves;
  int nrhs;
  const uint8_t *etype;
  const double *strains, *mats;
  double *out_stress, *out_strain;
  sp_solve_info *out_info, *task_info;
  unsigned *done;
  double rtol, inner_rtol;
  int max_outer, max_inner;
};

// The kernel class of an RVE (-1: none, the solve_rve kernel takes it)
int modes_class(const MeshGeo &g, const double *len, bool periodic, bool f64);
int modes_onchip(const MeshGeo &g, int threads, int room);
// Launches for the RVEs `ids` (largest first), every one of a class >= 0
int modes_plan(const std::vector<int> &ids, const std::vector<int> &cls,
               const std::vector<MeshGeo> &geo, int nrhs, bool periodic, bool f64, const Device *d,
               ModesPlan *out);
void modes_free(ModesPlan *m);
// counters: one per bucket, on the device
int modes_launch(const ModesPlan &m, const ModesCommon &c, int *counters,
                 cudaStream_t s, bool empty = false);

}  // namespace sp
