/*
 * model_check.cu - the integer forms that the step takes instead of the
 * model's comparisons and divisions (sampo_model.cuh), the functions
 * themselves against what they stand for.
 *
 *   model_check host     kill_threshold, as the host computes its tables
 *   model_check device   kill_threshold and the days of whole ages on a GPU
 */
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>
#include <vector>
#include "../sampo_gb300/csrc/sampo_model.cuh"

using namespace sampo;

// (float)v * 2^-32 <= hmr exactly for v < kill_threshold(hmr): at the
// threshold, beside it, and at the draws whose rounding is next to it.
__host__ __device__ static uint32_t threshold_fails(float hmr) {
  const uint32_t t = kill_threshold(hmr);
  const int64_t step[] = {0, 1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257, 600, 1 << 20};
  uint32_t bad = 0;
  for (int64_t d : step)
    for (int s = -1; s <= 1; s += 2) {
      const int64_t v = (int64_t)t + s * d;
      if (v < 0 || v > 0xffffffffll) continue;
      const bool dies = 2.3283064365387e-10f * (float)(uint32_t)v <= hmr;
      bad += dies != ((uint32_t)v < t);
    }
  return bad;
}
// Every `stride`-th float in [0, 0.98), and what is no mortality.
constexpr uint32_t kTop = 0x3f7ae148u;  // 0.98f

__global__ void k_check(uint32_t stride, uint32_t* bad) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
  uint32_t fails = 0;
  for (uint64_t j = (uint64_t)tid * stride; j < kTop; j += (uint64_t)n * stride) fails += threshold_fails(__uint_as_float((uint32_t)j)) != 0u;
  if (fails) atomicAdd(bad, fails);
  fails = 0;
  for (uint32_t h = tid; h < (1u << 21); h += n) {  // every whole age of a narrow pool
    const float age = (float)h;
    const uint32_t days = (uint32_t)(age / 24.0f);
    fails += whole_age_days(age) != days;
    fails += age_days<true>(age) != (days < 99u ? days : 99u) || age_days<true>(age) != age_days<false>(age);
    fails += age_days_uncapped<true>(age) != age_days_uncapped<false>(age);
    // as the larvae that stay have them: from one quotient, now and an hour on
    fails += whole_days(whole_age_quotient(age)) != days;
    fails += whole_days_next(whole_age_quotient(age)) != (uint32_t)((age + 1.0f) / 24.0f);
  }
  if (fails) atomicAdd(bad + 1, fails);
}

int main(int argc, char** argv) {
  uint32_t bad[2] = {0, 0};
  if (argc > 1 && !strcmp(argv[1], "device")) {
    uint32_t* d = nullptr;
    if (cudaMalloc(&d, sizeof(bad)) != cudaSuccess || cudaMemset(d, 0, sizeof(bad)) != cudaSuccess) return 2;
    k_check<<<304, 256>>>(3, d);
    if (cudaMemcpy(bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(d);
  } else {
    for (uint64_t j = 0; j < kTop; j += 251) {
      float h;
      const uint32_t w = (uint32_t)j;
      memcpy(&h, &w, 4);
      bad[0] += threshold_fails(h) != 0u;
    }
    for (int e = 1; e <= 40; e++) bad[0] += threshold_fails(1.0f / (float)(1ull << e)) != 0u;
    bad[0] += kill_threshold(0.0f / 0.0f * 0.0f) != 0u || kill_threshold(-1.0f) != 0u || kill_threshold(0.0f) != 1u;
  }
  printf("thresholds %u days %u\n", bad[0], bad[1]);
  return bad[0] || bad[1] ? 1 : 0;
}
