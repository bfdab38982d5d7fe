// sampo_kernels.cu - host side of the step kernels: grid sizes, launchers
// and the grid autotuner. The device code is in sampo_step_kernels.cuh.
#include <cuda_runtime.h>
#include <mutex>
#include <vector>
#include "sampo_step_kernels.cuh"
#include "sampo_small_step.cuh"

namespace sampo {

// ------------------------------------------------------------------------
// The built-in count and update/scatter passes for `items` rows at once.
// (the passes for whole records come with 4 only)
static const void* count_fn(int items, bool wide) {
  return wide ? (const void*)k_count<4, true> : items == 2 ? (const void*)k_count<2, false> : (const void*)k_count<4, false>;
}
static const void* scatter_fn(int items, bool wide, bool ahead = false) {
  if (wide) return (const void*)k_scatter<4, true, false>;
  if (ahead) return items == 2 ? (const void*)k_scatter<2, false, true> : (const void*)k_scatter<4, false, true>;
  return items == 2 ? (const void*)k_scatter<2, false, false> : (const void*)k_scatter<4, false, false>;
}

// The SM count of the current device, after its one-time set-up: the dynamic
// shared memory limit of the two passes (a function attribute applies to the
// device that is current when it is set, so every device the library runs on
// gets its own; devices beyond kMaxDevices are set up on every call).
static int setup_device(int dev) {
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  const int smem = (int)pass_smem(kMaxRep);
  for (int items : {2, 4})
    for (bool wide : {false, true}) {
      cudaFuncSetAttribute(count_fn(items, wide), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      for (bool ahead : {false, true})
        cudaFuncSetAttribute(scatter_fn(items, wide, ahead), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    }
  return n > 0 ? n : 1;
}
static int sm_count() {
  constexpr int kMaxDevices = 64;
  static std::once_flag once[kMaxDevices];
  static int sms[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDevices) return setup_device(dev);
  std::call_once(once[dev], [&] { sms[dev] = setup_device(dev); });
  return sms[dev];
}
int device_sms() { return sm_count(); }
size_t pass_smem_max() { return pass_smem(kMaxRep); }

// Resident CTAs per SM of a pass, built in or of ks (4 rows at once).
static int occupancy(const void* ks, bool scatter, int items, bool wide, uint32_t nrep) {
  if (ks)
    return species_occupancy(ks, scatter ? (wide ? KID_SCATTER_WIDE : KID_SCATTER) : (wide ? KID_COUNT_WIDE : KID_COUNT), kBlock,
                             pass_smem(nrep));
  (void)sm_count();  // the set-up
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, scatter ? scatter_fn(items, wide) : count_fn(items, wide), kBlock,
                                                pass_smem(nrep));
  return per;
}
int grid_blocks_count(uint32_t nrep, const void* ks, int items, bool wide) {
  const int per = occupancy(ks, false, items, wide, nrep);
  return sm_count() * (per > 0 ? per : 1);
}
int grid_blocks_scatter(uint32_t nrep, const void* ks, int items, bool wide) {
  const int per = occupancy(ks, true, items, wide, nrep);
  return sm_count() * (per > 0 ? per : 1);
}

// One launch of kernel kid: the built-in one (fn) or p.ks's. `early`: a kernel
// that waits for the one before itself (wait_previous_kernel); launched so in
// batches only, where the passes' prologue scans the replicates (96
// replicates for 20 days: 110.5 ms without, 107.3 with; 1e6 eggs for two
// months alone: 171.8 without, 172.5 with).
static cudaError_t launch(const KParams& p, int kid, const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                          void** args, bool early = false) {
  if (p.ks) return species_launch(p.ks, kid, grid, block, smem, st, args);
  (void)sm_count();  // the set-up
  if (early && p.nrep > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
  }
  return cudaLaunchKernel(fn, grid, block, args, smem, st);
}

cudaError_t launch_count(const KParams& p, int grid, cudaStream_t st, int items) {
  KParams q = p;
  void* args[] = {&q};
  return launch(p, p.wide ? KID_COUNT_WIDE : KID_COUNT, count_fn(items, p.wide), grid, kBlock, pass_smem(p.nrep), st, args,
                true);
}
cudaError_t launch_scatter(const KParams& p, int grid, cudaStream_t st, int items, bool ahead) {
  KParams q = p;
  void* args[] = {&q};
  return launch(p, p.wide ? KID_SCATTER_WIDE : KID_SCATTER, scatter_fn(items, p.wide, ahead), grid, kBlock, pass_smem(p.nrep), st,
                args, true);
}
cudaError_t launch_steps(const KParams& p, uint32_t nsteps, bool ahead, int grid_count, int grid_scatter, int items, cudaStream_t st,
                         uint32_t* launches) {
  cudaError_t e = cudaSuccess;
  uint32_t n = 0;
  auto run = [&](cudaError_t x) {
    e = x;
    n++;
    return x == cudaSuccess;
  };
  if (ahead && can_decide_ahead(p) && nsteps > 1) {
    // one count pass; every pass but the last decides the hour after its own
    bool ok = run(launch_count(p, grid_count, st, items)) && run(launch_publish(p, PUB_DECIDED | PUB_AHEAD, st));
    for (uint32_t i = 0; i < nsteps && ok; i++)
      ok = run(launch_scatter(p, grid_scatter, st, items, i + 1 < nsteps)) &&
           run(launch_publish(p, PUB_AFTER_STEP | (i + 2 < nsteps ? PUB_AHEAD : 0), st));
  } else {
    for (uint32_t i = 0; i < nsteps; i++)
      if (!run(launch_count(p, grid_count, st, items)) || !run(launch_scatter(p, grid_scatter, st, items, false)) ||
          !run(launch_publish(p, PUB_AFTER_STEP, st)))
        break;
  }
  if (launches) *launches += n;
  return e;
}
cudaError_t launch_publish(const KParams& p, int mode, cudaStream_t st) {
  KParams q = p;
  void* args[] = {&q, &mode};
  return launch(p, KID_PUBLISH, (const void*)k_publish, p.nrep, mode == PUB_REFRESH ? 32 : kPublishThreads, 0, st, args,
                mode != PUB_REFRESH);
}
cudaError_t launch_init_eggs(const KParams& p, uint32_t n, float T0, const sampo_seeds* seeds_dev, int age_days_max,
                             uint64_t age_seed, bool full, cudaStream_t st) {
  KParams q = p;
  int fc = full ? 1 : 0;
  void* args[] = {&q, &n, &T0, &seeds_dev, &age_days_max, &age_seed, &fc};
  return launch(p, KID_INIT_EGGS, (const void*)k_init_eggs, sm_count() * 4, 256, 0, st, args);
}
cudaError_t launch_begin_step(const KParams& p, const CtxInputs& in, uint32_t slot, cudaStream_t st) {
  KParams q = p;
  CtxInputs x = in;
  void* args[] = {&q, &x, &slot};
  return launch(p, KID_BEGIN_STEP, (const void*)k_begin_step, 1, 32, 0, st, args);
}
cudaError_t launch_publish_start(const KParams& p, uint32_t flags, uint32_t end, cudaStream_t st) {
  KParams q = p;
  void* args[] = {&q, &flags};
  // four slots a thread and turn; a small pool gets no more CTAs than that takes (their start is most of its time)
  const int grid = (int)std::min((uint64_t)sm_count() * 4, std::max<uint64_t>(units_of(end, 1024), 1));
  cudaError_t e = launch(p, KID_POOL_STATS, (const void*)k_pool_stats, grid, 256, 0, st, args);
  if (e != cudaSuccess) return e;
  int mode = PUB_INITIAL;
  void* args2[] = {&q, &mode};
  return launch(p, KID_PUBLISH, (const void*)k_publish, 1, kPublishThreads, 0, st, args2);
}
cudaError_t launch_widen(const KParams& p, cudaStream_t st) {
  KParams q = p;
  void* args[] = {&q};
  return launch(p, KID_WIDEN, (const void*)k_widen, sm_count() * 4, 256, 0, st, args);
}
cudaError_t launch_histogram(const KParams& p, uint32_t* hist_dev, cudaStream_t st) {
  KParams q = p;
  void* args[] = {&q, &hist_dev};
  return launch(p, KID_HISTOGRAM, (const void*)k_histogram, sm_count() * 4, 256, 0, st, args);
}
static cudaError_t launch_trial_reset(const KParams& p, cudaStream_t st) {
  KParams q = p;
  void* args[] = {&q};
  return launch(p, KID_TRIAL_RESET, (const void*)k_trial_reset, (int)((p.nrep + 255) / 256), 256, 0, st, args);
}
// The grid tuner of one number of rows at once: see tune_grids.
static cudaError_t tune_grids_items(const KParams& p, cudaStream_t st, int items, cudaEvent_t* ev, int* grid_count,
                                    int* grid_scatter, double* best_ms) {
  int max_c = occupancy(p.ks, false, items, p.wide, p.nrep);
  int max_s = occupancy(p.ks, true, items, p.wide, p.nrep);
  if (max_c < 1) max_c = 1;
  if (max_s < 1) max_s = 1;
  const int sms = sm_count();
  cudaError_t e = cudaSuccess;
  // each kernel's time is taken on its own (the best count grid does not
  // depend on the scatter grid), minimum over every trial that ran it (eight
  // per pair: small pools run the kernels in tens of microseconds, where
  // single timings differ by more than the grids do); one untimed trial first
  double tc[9], ts[9];
  for (int i = 0; i < 9; i++) tc[i] = ts[i] = 1e30;
  max_c = max_c > 8 ? 8 : max_c;
  max_s = max_s > 8 ? 8 : max_s;
  for (int c = 1; c <= max_c && e == cudaSuccess; c++) {
    for (int s = 1; s <= max_s && e == cudaSuccess; s++) {
      for (int rep = (c == 1 && s == 1) ? -1 : 0; rep < 8 && e == cudaSuccess; rep++) {
        if ((e = launch_trial_reset(p, st)) != cudaSuccess) break;
        if ((e = cudaEventRecord(ev[0], st)) != cudaSuccess) break;
        if ((e = launch_count(p, c * sms, st, items)) != cudaSuccess) break;
        if ((e = cudaEventRecord(ev[1], st)) != cudaSuccess) break;
        if ((e = launch_scatter(p, s * sms, st, items)) != cudaSuccess) break;
        if ((e = cudaEventRecord(ev[2], st)) != cudaSuccess) break;
        if ((e = cudaEventSynchronize(ev[2])) != cudaSuccess) break;
        if (rep < 0) continue;
        float m0 = 0, m1 = 0;
        cudaEventElapsedTime(&m0, ev[0], ev[1]);
        cudaEventElapsedTime(&m1, ev[1], ev[2]);
        if (m0 < tc[c]) tc[c] = m0;
        if (m1 < ts[s]) ts[s] = m1;
      }
    }
  }
  int bc = max_c, bs = max_s;
  for (int c = 1; c <= max_c; c++)
    if (tc[c] < tc[bc]) bc = c;
  for (int s = 1; s <= max_s; s++)
    if (ts[s] < ts[bs]) bs = s;
  // the kernels run back to back in a step, where a small pool's times are
  // mostly start-up and tail: the pick and the largest grids, run that way
  double tj[2] = {1e30, 1e30};
  const int gc[2] = {bc, max_c}, gs[2] = {bs, max_s};
  for (int rep = 0; rep < 8 && e == cudaSuccess; rep++) {
    for (int v = 0; v < 2 && e == cudaSuccess; v++) {
      if (v == 1 && bc == max_c && bs == max_s) break;
      if ((e = launch_trial_reset(p, st)) != cudaSuccess) break;
      if ((e = cudaEventRecord(ev[0], st)) != cudaSuccess) break;
      if ((e = launch_count(p, gc[v] * sms, st, items)) != cudaSuccess) break;
      if ((e = launch_scatter(p, gs[v] * sms, st, items)) != cudaSuccess) break;
      if ((e = cudaEventRecord(ev[2], st)) != cudaSuccess) break;
      if ((e = cudaEventSynchronize(ev[2])) != cudaSuccess) break;
      float m = 0;
      cudaEventElapsedTime(&m, ev[0], ev[2]);
      if (m < tj[v]) tj[v] = m;
    }
  }
  if (bc != max_c || bs != max_s) {
    if (tj[1] <= tj[0]) {
      bc = max_c;
      bs = max_s;
      tj[0] = tj[1];
    }
  }
  *grid_count = bc * sms;
  *grid_scatter = bs * sms;
  *best_ms = tj[0];
  return e;
}

cudaError_t tune_grids(const KParams& p, cudaStream_t st, int* grid_count, int* grid_scatter, int* items, double* best_ms) {
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 3 && e == cudaSuccess; i++) e = cudaEventCreate(&ev[i]);
  // 4 rows at once and, for the built-in species, 2; the step as a whole decides
  double best = 1e30;
  int bi = kItems, bgc = 0, bgs = 0;
  for (int it : {4, 2}) {
    if (e != cudaSuccess || (it != kItems && p.ks)) break;
    int gc = 0, gs = 0;
    double ms = 1e30;
    e = tune_grids_items(p, st, it, ev, &gc, &gs, &ms);
    if (e == cudaSuccess && ms < best) {
      best = ms;
      bi = it;
      bgc = gc;
      bgs = gs;
    }
  }
  if (e == cudaSuccess) e = launch_trial_reset(p, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  for (int i = 0; i < 3; i++)
    if (ev[i]) cudaEventDestroy(ev[i]);
  *grid_count = bgc;
  *grid_scatter = bgs;
  *items = bi;
  if (best_ms) *best_ms = best;
  return e;
}
static int small_kid(int items) { return items == 1 ? KID_SMALL1 : items == 2 ? KID_SMALL2 : KID_SMALL4; }
static const void* small_fn(int items) {
  return items == 1 ? (const void*)k_step_small<1> : items == 2 ? (const void*)k_step_small<2> : (const void*)k_step_small<4>;
}
int grid_blocks_small(int items, const void* ks) {
  int per = 0;
  if (ks) return sm_count() * species_occupancy(ks, small_kid(items), kSmallThreads, small_stage(items));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, small_fn(items), kSmallThreads, small_stage(items)) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return sm_count() * per;
}

int grid_blocks_small_all(const void* ks) {
  return std::min({grid_blocks_small(1, ks), grid_blocks_small(2, ks), grid_blocks_small(4, ks)});
}
cudaError_t launch_small_hour(const KParams& p, uint32_t end, int items, int max_grid, cudaStream_t st) {
  const uint64_t want = (uint64_t)units_of(end, (uint32_t)(kBlock * items)) + 1u;
  return launch_small(p, (int)std::min(want, (uint64_t)max_grid), true, 1u, st, items);
}

cudaError_t graph_kernel_nodes(cudaGraph_t g, uint32_t* kernels) {
  size_t nn = 0;
  cudaError_t e = cudaGraphGetNodes(g, nullptr, &nn);
  std::vector<cudaGraphNode_t> nodes(nn);
  if (e == cudaSuccess && nn) e = cudaGraphGetNodes(g, nodes.data(), &nn);
  uint32_t k = 0;
  for (size_t i = 0; i < nn && e == cudaSuccess; i++) {
    cudaGraphNodeType t;
    e = cudaGraphNodeGetType(nodes[i], &t);
    k += t == cudaGraphNodeTypeKernel ? 1u : 0u;
  }
  *kernels = k;
  return e;
}

cudaError_t launch_small(const KParams& p, int grid, bool cooperative, uint32_t nsteps, cudaStream_t st, int items) {
  KParams q = p;
  void* args[] = {&q, &nsteps};
  if (p.ks)
    return species_launch(p.ks, small_kid(items), dim3(grid), dim3(kSmallThreads), small_stage(items), st, args, cooperative);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kSmallThreads);
  cfg.dynamicSmemBytes = small_stage(items);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cooperative ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, small_fn(items), args);
}
// What a server asks of every slot, 16 bytes each: step, active, status bits
// and pool end. (The strided copy of the states' heads, 1024 x 0.5 KB to
// pageable memory, took 0.14 ms per call, this 0.025.)
__global__ void k_slot_states(const SimDev* sims, uint32_t n, uint4* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = make_uint4(sims[i].step, sims[i].active, sims[i].error | sims[i].warn, sims[i].pop.r[GRAVID].end);
}
cudaError_t launch_slot_states(const SimDev* sims, uint32_t n, uint4* out, cudaStream_t st) {
  k_slot_states<<<(n + 127u) / 128u, 128, 0, st>>>(sims, n, out);
  return cudaGetLastError();
}
cudaError_t launch_eval_math(int fn, const float* x, const float* y, float* out, uint32_t n, cudaStream_t st) {
  k_eval_math<<<sm_count() * 2, 256, 0, st>>>(fn, x, y, out, n);
  return cudaGetLastError();
}

}  // namespace sampo
