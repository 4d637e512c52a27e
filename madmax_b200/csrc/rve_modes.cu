// rve_modes.cu -- host side of the element-mode batch kernel.
#include <algorithm>

#include "rve_modes_host.h"

namespace sp {

SP_MODES_CLASSES(SP_MODES_EXTERN, F2, false)
SP_MODES_CLASSES(SP_MODES_EXTERN, F2, true)
SP_MODES_CLASSES(SP_MODES_EXTERN, double, false)
SP_MODES_CLASSES(SP_MODES_EXTERN, double, true)
SP_MODES_PERIODIC(SP_MODES_EXTERN, F2)
SP_MODES_PERIODIC(SP_MODES_EXTERN, double)
SP_MODES_AFFINE(SP_MODES_EXTERN, F2)
SP_MODES_AFFINE(SP_MODES_EXTERN, double)

struct ModesClass {
  int threads, minb, on;
  ModesFn fn[2][2][2];  // [FP64][periodic][cubes]
};

#define SP_MODES_FNS(V, NT, MINB, ON, PER) \
  {k_modes<V, NT, MINB, false, ON, PER>, k_modes<V, NT, MINB, true, ON, PER>}
#define SP_MODES_ROW(V, NT, MINB, ON, PER) \
  {NT, MINB, ON, \
   {{SP_MODES_FNS(F2, NT, MINB, ON, false), SP_MODES_FNS(F2, NT, MINB, ON, true)}, \
    {SP_MODES_FNS(double, NT, MINB, ON, false), SP_MODES_FNS(double, NT, MINB, ON, true)}}},
static const ModesClass kClasses[] = {
    SP_MODES_CLASSES(SP_MODES_ROW, F2, false)
    {640, 1, 1,
     {{{nullptr, nullptr}, SP_MODES_FNS(F2, 640, 1, 1, true)},
      {{nullptr, nullptr}, SP_MODES_FNS(double, 640, 1, 1, true)}}},
    {512, 1, 0,
     {{SP_MODES_FNS(F2, 512, 1, 0, false), {nullptr, nullptr}},
      {SP_MODES_FNS(double, 512, 1, 0, false), {nullptr, nullptr}}}},
};
#undef SP_MODES_ROW
#undef SP_MODES_FNS
constexpr int kNumClasses = sizeof(kClasses) / sizeof(kClasses[0]);

// shared memory of one SM and what a block holds beside its dynamic part
constexpr int SP_MODES_SM_BYTES = 228 * 1024, SP_MODES_BLOCK_MAX = 227 * 1024;
constexpr int SP_MODES_RESERVED = 1024;

// dynamic shared memory a CTA of a class may use
static int class_room(const ModesClass &k) {
  return (std::min(SP_MODES_SM_BYTES / k.minb, SP_MODES_BLOCK_MAX + 1024) - SP_MODES_RESERVED) / 16 * 16;
}

// The vectors a CTA of `threads` threads and `room` bytes of dynamic shared
// memory keeps there for an affine FP32 RVE (-1: none of the element-mode kernels)
int modes_onchip(const MeshGeo &g, int threads, int room) {
  if (g.nex < 2 || g.ney < 2 || g.nez < 2 || g.nez > SP_MODES_MAX_NEZ) return -1;
  if ((long long)g.nex * g.ney > SP_MODES_MAX_COLS) return -1;
  for (int on = 2; on >= 0; on--) {
    const ModesGeo G(g.nex, g.ney, g.nez, false, false, on);
    if (G.rows >= 1 && G.warps() * 32 <= threads && G.smem() <= room) return on;
  }
  return -1;
}

// An RVE runs on the smallest class whose threads hold one element column
// each and whose shared memory holds its vectors beside the
// class's other CTAs; it needs an interior node on every axis, at most 32
// element layers, 30 under periodic conditions (a column's materials are one
// 32-bit mask, which repeats two layers then), and at most 1024 columns.
// Larger RVEs keep the solve_rve kernel.
int modes_class(const MeshGeo &g, const double *len, bool per, bool f64) {
  if (g.nex < 2 || g.ney < 2 || g.nez < 2) return -1;
  if (g.nez > (per ? SP_MODES_MAX_NEZ - 2 : SP_MODES_MAX_NEZ)) return -1;
  if ((long long)g.nex * g.ney > SP_MODES_MAX_COLS) return -1;
  const double hx = len[0] / g.nex, hy = len[1] / g.ney, hz = len[2] / g.nez;
  const int cube = hx == hy && hx == hz;
  for (int c = 0; c < kNumClasses; c++) {
    const ModesClass &k = kClasses[c];
    if (!k.fn[f64][per][cube]) continue;
    const ModesGeo G(g.nex, g.ney, g.nez, per, f64, k.on);
    if (G.rows >= 1 && G.warps() * 32 <= k.threads && G.smem() <= class_room(k)) return 2 * c + cube;
  }
  return -1;
}

int modes_plan(const std::vector<int> &ids, const std::vector<int> &cls,
               const std::vector<MeshGeo> &geo, int nrhs, bool per, bool f64, const Device *d,
               ModesPlan *out) {
  // classes with the largest RVEs first
  for (int c = 2 * kNumClasses - 1; c >= 0; c--) {
    std::vector<int> ord;
    for (int i : ids)
      if (cls[i] == c) ord.push_back(i);
    if (ord.empty()) continue;
    const ModesClass &k = kClasses[c / 2];
    out->buckets.push_back(ModesBucket());
    ModesBucket &b = out->buckets.back();
    b.fn = k.fn[f64][per][c & 1];
    b.nrve = (int)ord.size();
    int ntot = 0, wlen = 0, elen = 0;
    for (int i : ord) {
      const ModesGeo G(geo[i].nex, geo[i].ney, geo[i].nez, per, f64, k.on);
      b.threads = std::max(b.threads, G.warps() * 32);
      b.smem = std::max(b.smem, G.smem());
      ntot = std::max(ntot, G.ntot);
      wlen = std::max(wlen, G.wlen());
      elen = std::max(elen, 6 * G.mz * G.nex);
    }
    b.w_stride = ((size_t)3 * wlen + 15) / 16 * 16;
    b.v_stride = ((size_t)3 * ntot + 15) / 16 * 16;
    b.v_cta = (size_t)(4 - k.on) * b.v_stride;
    // the class's largest, the same for every batch: the attribute is the
    // function's, not the launch's
    if (cudaFuncSetAttribute((const void *)b.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             class_room(k)) != cudaSuccess) {
      cudaGetLastError();
      return sp_set_error(SP_ERR_CUDA, "sp_batch_create: %d bytes of dynamic shared memory refused",
                          class_room(k));
    }
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, (const void *)b.fn, b.threads, b.smem) !=
            cudaSuccess ||
        nb < 1) {
      cudaGetLastError();
      return sp_set_error(SP_ERR_CUDA, "sp_batch_create: %d-thread CTAs cannot be resident", b.threads);
    }
    b.grid = (int)std::min<long long>((long long)d->nsm * nb, (long long)b.nrve * nrhs);
    SP_TRY(dmalloc((void **)&b.d_order, ord.size() * sizeof(int), &b.bytes));
    SP_TRY(dmalloc((void **)&b.ws_w, b.grid * b.w_stride * sizeof(double), &b.bytes));
    SP_TRY(dmalloc((void **)&b.ws_v, b.grid * b.v_cta * sizeof(double), &b.bytes));
    if (k.on < 2) {
      b.e_stride = ((size_t)elen + 15) / 16 * 16;
      SP_TRY(dmalloc((void **)&b.ws_e, b.grid * b.e_stride * sizeof(double), &b.bytes));
    }
    if (cudaMemcpy(b.d_order, ord.data(), ord.size() * sizeof(int), cudaMemcpyHostToDevice))
      return sp_set_error(SP_ERR_CUDA, "sp_batch_create: upload failed");
  }
  for (size_t i = 1; i < out->buckets.size(); i++) {
    cudaStream_t st;
    cudaEvent_t ev;
    SP_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    out->side.push_back(st);
    SP_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    out->joined.push_back(ev);
  }
  if (!out->side.empty())
    SP_CUDA_TRY(cudaEventCreateWithFlags(&out->forked, cudaEventDisableTiming));
  return SP_OK;
}

void modes_free(ModesPlan *m) {
  for (ModesBucket &k : m->buckets) {
    cudaFree(k.d_order);
    cudaFree(k.ws_w);
    cudaFree(k.ws_v);
    cudaFree(k.ws_e);
  }
  for (cudaStream_t s : m->side) cudaStreamDestroy(s);
  for (cudaEvent_t e : m->joined) cudaEventDestroy(e);
  if (m->forked) cudaEventDestroy(m->forked);
  *m = ModesPlan();
}

int modes_launch(const ModesPlan &m, const ModesCommon &c, int *counters, cudaStream_t s,
                 bool empty) {
  const std::vector<ModesBucket> &b = m.buckets;
  if (b.empty()) return SP_OK;
  SP_CUDA_TRY(cudaMemsetAsync(counters, 0, b.size() * sizeof(int), s));
  if (b.size() > 1) SP_CUDA_TRY(cudaEventRecord(m.forked, s));
  for (size_t i = 0; i < b.size(); i++) {
    const ModesBucket &k = b[i];
    ModesParams P;
    P.plans = c.plans;
    P.rves = c.rves;
    P.order = k.d_order;
    P.nrhs = c.nrhs;
    P.ntask = empty ? 0 : k.nrve * c.nrhs;
    P.etype = c.etype;
    P.strains = c.strains;
    P.mats = c.mats;
    P.out_stress = c.out_stress;
    P.out_strain = c.out_strain;
    P.out_info = c.out_info;
    P.task_info = c.task_info;
    P.done = c.done;
    P.counter = counters + i;
    P.buf = ModesBufs{k.ws_w, k.ws_v, k.ws_e, k.w_stride, k.v_stride, k.e_stride, k.v_cta};
    P.lim = ModesLimits{c.rtol, c.inner_rtol, c.rtol, c.max_outer, c.max_inner};
    cudaStream_t st = i ? m.side[i - 1] : s;
    if (i) SP_CUDA_TRY(cudaStreamWaitEvent(st, m.forked, 0));
    k.fn<<<k.grid, k.threads, k.smem, st>>>(P);
    SP_CUDA_TRY(cudaGetLastError());
    if (i) SP_CUDA_TRY(cudaEventRecord(m.joined[i - 1], st));
  }
  for (size_t i = 1; i < b.size(); i++) {
    SP_CUDA_TRY(cudaStreamWaitEvent(s, m.joined[i - 1], 0));
  }
  return SP_OK;
}

}  // namespace sp
