/*
 * fake_cuda.h - a CUDA runtime in host memory and the kernel launchers of the
 * library as counters, so that the host side of the C ABI runs without a GPU
 * and a test can give it any device state or refuse any launch. Included by
 * one host_*_check.cu, before the source file of the library that it checks.
 *
 * "Device" memory is malloc'd memory, so a check reads and writes a
 * simulation's device state directly; streams are synchronous.
 */
#pragma once
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include "../sampo_gb300/csrc/sampo_model.cuh"
#include "../sampo_gb300/csrc/sampo_kernels.cuh"

static int g_checks_failed = 0;
#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      printf("%s:%d: %s\n", __FILE__, __LINE__, #x);          \
      g_checks_failed++;                                      \
    }                                                         \
  } while (0)

// What the launchers were asked for, and what the next of them answers.
static std::map<std::string, int> g_launches;
static cudaError_t g_small_answer = cudaSuccess;  // launch_small, launch_small_hour
static int g_resident = 3;                        // CTAs per SM of narrow passes
static int g_resident_wide = 3;                   // and of wide ones
static uint32_t g_wide_found = 0;                 // what launch_publish_start's check finds
constexpr int kFakeSms = 10;

static inline cudaError_t fake_cudaSetDevice(int) { return cudaSuccess; }
static inline cudaError_t fake_cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
static inline cudaError_t fake_cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? kFakeSms : 1 << 20; return cudaSuccess; }
template <class T>
static inline cudaError_t fake_cudaMalloc(T** p, size_t n) { *p = (T*)malloc(n ? n : 1); memset(*p, 0xA5, n); return cudaSuccess; }
template <class T>
static inline cudaError_t fake_cudaMallocHost(T** p, size_t n) { return fake_cudaMalloc(p, n); }
static inline cudaError_t fake_cudaFree(void* p) { free(p); return cudaSuccess; }
static inline cudaError_t fake_cudaFreeHost(void* p) { free(p); return cudaSuccess; }
static inline cudaError_t fake_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake_cudaMalloc(p, n); }
static inline cudaError_t fake_cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
static inline cudaError_t fake_cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
static inline cudaError_t fake_cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
static inline cudaError_t fake_cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memmove(d, s, n); return cudaSuccess; }
static inline cudaError_t fake_cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memmove(d, s, n); return cudaSuccess; }
static inline cudaError_t fake_cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t i = 0; i < h; i++) memmove((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
static inline cudaError_t fake_cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
static inline cudaError_t fake_cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
static inline cudaError_t fake_cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
static inline cudaError_t fake_cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
static inline cudaError_t fake_cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
static inline cudaError_t fake_cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = (cudaGraphExec_t)malloc(1); return cudaSuccess; }
static inline cudaError_t fake_cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { g_launches["graph"]++; return cudaSuccess; }
static inline cudaError_t fake_cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
static inline cudaError_t fake_cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
static inline cudaError_t fake_cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
static inline cudaError_t fake_cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
static inline cudaError_t fake_cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
alignas(256) static unsigned char g_fake_symbol[32u << 20];  // the one __device__ array of the library
template <class T>
static inline cudaError_t fake_cudaGetSymbolAddress(void** p, const T& t) {
  *p = g_fake_symbol;
  return sizeof(t) <= sizeof(g_fake_symbol) ? cudaSuccess : cudaErrorInvalidSymbol;
}
static inline cudaError_t fake_cudaGetLastError(void) { return cudaSuccess; }
static inline const char* fake_cudaGetErrorString(cudaError_t) { return "fake"; }
#define cudaSetDevice fake_cudaSetDevice
#define cudaGetDevice fake_cudaGetDevice
#define cudaDeviceGetAttribute fake_cudaDeviceGetAttribute
#define cudaMalloc fake_cudaMalloc
#define cudaMallocHost fake_cudaMallocHost
#define cudaFree fake_cudaFree
#define cudaFreeHost fake_cudaFreeHost
#define cudaMallocFromPoolAsync fake_cudaMallocFromPoolAsync
#define cudaFreeAsync fake_cudaFreeAsync
#define cudaMemPoolCreate fake_cudaMemPoolCreate
#define cudaMemPoolDestroy fake_cudaMemPoolDestroy
#define cudaMemPoolSetAttribute fake_cudaMemPoolSetAttribute
#define cudaMemcpy fake_cudaMemcpy
#define cudaMemcpyAsync fake_cudaMemcpyAsync
#define cudaMemcpy2DAsync fake_cudaMemcpy2DAsync
#define cudaMemsetAsync fake_cudaMemsetAsync
#define cudaStreamCreateWithFlags fake_cudaStreamCreateWithFlags
#define cudaStreamDestroy fake_cudaStreamDestroy
#define cudaStreamSynchronize fake_cudaStreamSynchronize
#define cudaStreamIsCapturing fake_cudaStreamIsCapturing
#define cudaStreamBeginCapture fake_cudaStreamBeginCapture
#define cudaStreamEndCapture fake_cudaStreamEndCapture
#define cudaGraphInstantiate fake_cudaGraphInstantiate
#define cudaGraphLaunch fake_cudaGraphLaunch
#define cudaGraphExecDestroy fake_cudaGraphExecDestroy
#define cudaGraphDestroy fake_cudaGraphDestroy
#define cudaEventCreate fake_cudaEventCreate
#define cudaEventCreateWithFlags fake_cudaEventCreateWithFlags
#define cudaEventDestroy fake_cudaEventDestroy
#define cudaEventRecord fake_cudaEventRecord
#define cudaEventSynchronize fake_cudaEventSynchronize
#define cudaEventElapsedTime fake_cudaEventElapsedTime
#define cudaGetSymbolAddress fake_cudaGetSymbolAddress
#define cudaGetLastError fake_cudaGetLastError
#define cudaGetErrorString fake_cudaGetErrorString

extern "C" int sampo_species_device(const sampo_species*) { return 0; }

namespace sampo {
static cudaError_t note(const char* what) { g_launches[what]++; return cudaSuccess; }
int grid_blocks_count(uint32_t, const void*, int, bool wide) { return kFakeSms * (wide ? g_resident_wide : g_resident); }
int grid_blocks_scatter(uint32_t, const void*, int, bool wide) { return kFakeSms * (wide ? g_resident_wide : g_resident); }
int device_sms() { return kFakeSms; }
int grid_blocks_small_all(const void*) { return kFakeSms * 3; }
cudaError_t launch_count(const KParams& p, int, cudaStream_t, int) {
  const uint32_t n = units_of(span_count(p.reps[0].sim->pop.r[7].end, 0), 32) * 4, *w = reinterpret_cast<const uint32_t*>(p.reps[0].supers);
  bool clean = true;
  for (uint32_t i = 0; i < n; i++) clean &= w[i] == 0;
  if (clean) note("count on clean supers");
  return note("count");
}
cudaError_t launch_scatter(const KParams&, int, cudaStream_t, int, bool) { return note("scatter"); }
cudaError_t launch_steps(const KParams& p, uint32_t n, bool, int, int, int, cudaStream_t, uint32_t* launches) {
  if (launches) *launches += 3 * n;
  p.reps[0].sim->step += n;
  return note("steps");
}
cudaError_t launch_publish(const KParams&, int, cudaStream_t) { return note("publish"); }
cudaError_t launch_init_eggs(const KParams&, uint32_t, float, const sampo_seeds*, int, uint64_t, bool full, cudaStream_t) {
  return note(full ? "init, whole" : "init");
}
cudaError_t launch_publish_start(const KParams& p, uint32_t flags, uint32_t, cudaStream_t) {
  if (flags & PS_CHECK) p.reps[0].sim->wide = g_wide_found;
  if (flags & PS_CLEAR) memset(p.reps[0].supers, 0, units_of(span_count(p.reps[0].sim->pop.r[7].end, 0), 32) * sizeof(uint4));
  if (flags & PS_ROWS) memset(p.reps[0].smallRows, 0, small_row_words(p.reps[0].smallTiles) * 4);
  return note("start");
}
cudaError_t launch_begin_step(const KParams&, const CtxInputs&, uint32_t, cudaStream_t) { return note("begin"); }
cudaError_t launch_widen(const KParams&, cudaStream_t) { return note("widen"); }
cudaError_t launch_histogram(const KParams&, uint32_t*, cudaStream_t) { return note("histogram"); }
cudaError_t launch_slot_states(const SimDev* sims, uint32_t n, uint4* out, cudaStream_t) {
  for (uint32_t i = 0; i < n; i++) out[i] = make_uint4(sims[i].step, sims[i].active, sims[i].error | sims[i].warn, sims[i].pop.r[7].end);
  return cudaSuccess;
}
cudaError_t launch_eval_math(int, const float*, const float*, float*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t graph_kernel_nodes(cudaGraph_t, uint32_t* k) { *k = 1; return cudaSuccess; }
static cudaError_t note_small(const KParams& p, const char* what) {
  const RepParams& rp = p.reps[0];
  bool clean = p.bat->bar == 0 && p.bat->done == 0;
  for (size_t i = 0; i < small_row_words(rp.smallTiles); i++)  // (the tiles' words between are written before they are read)
    clean &= rp.smallRows[i] == 0 || (i >= small_group_words(rp.smallTiles) && i < small_row_words(rp.smallTiles) - 4);
  note(what);
  if (clean) note("small on clean rows");
  return g_small_answer;
}
cudaError_t launch_small_hour(const KParams& p, uint32_t, int, int, cudaStream_t) { return note_small(p, "small"); }
cudaError_t launch_small(const KParams& p, int, bool, uint32_t, cudaStream_t, int) { return note_small(p, "small day"); }
cudaError_t tune_grids(const KParams&, cudaStream_t, int* c, int* s, int* items, double*) {
  *c = 2 * kFakeSms;
  *s = kFakeSms;
  *items = 4;
  return cudaSuccess;
}
}  // namespace sampo
