/*
 * host_noalloc_check.cu - the host side of sampo_step_noalloc (sampo_noalloc.cu)
 * on fake_cuda.h.
 */
#include "fake_cuda.h"
#include "../sampo_gb300/csrc/sampo_noalloc.cu"

static int one_step(uint32_t eggs) {
  const uint32_t cap = 1u << 17;
  static unsigned char mem[2][10][(1u << 17) * 4 + 64];
  sampo_device_pool d[2];
  for (int k = 0; k < 2; k++) {
    void* c[10];
    for (int i = 0; i < 10; i++) c[i] = (void*)(((uintptr_t)mem[k][i] + 15) & ~(uintptr_t)15);
    d[k] = {(float*)c[0], (float*)c[1], (float*)c[2], (float*)c[3], (uint32_t*)c[4], (uint32_t*)c[5], (uint32_t*)c[6], (uint32_t*)c[7], (uint32_t*)c[8], (uint8_t*)c[9]};
  }
  sampo_population pop, out;
  memset(&pop, 0, sizeof(pop));
  pop.r[0].end = eggs;
  for (uint32_t k = 1; k < 8; k++) pop.r[k].start = pop.r[k].end = pop.r[k - 1].end + 64;
  sampo_environment env;
  memset(&env, 0, sizeof(env));
  env.carryingCapacity = 1000.0f;
  sampo_seeds seeds[4];
  memset(seeds, 0, sizeof(seeds));
  sampo_stats_row row;
  sampo_bites_cycles bnc;
  return sampo_step_noalloc(&d[0], cap, &d[1], cap, &pop, &env, 25.0f, 0, seeds, 1000.0f, &row, &out, &bnc, 0, nullptr);
}

// A refused cooperative launch: the passes step the hour, on cleared supers
// (the array keeps whatever the calls before left in it).
static void refused_launches_take_the_passes() {
  memset(((Scratch*)g_fake_symbol)->spans, 0x11, sizeof(Scratch::spans));
  g_small_answer = cudaErrorCooperativeLaunchTooLarge;
  g_launches.clear();
  CHECK(one_step(1000) == SAMPO_OK);
  CHECK(g_launches["small"] == 1 && g_launches["count"] == 1 && g_launches["scatter"] == 1 && g_launches["publish"] == 1);
  CHECK(g_launches["count on clean supers"] == 1);
  g_small_answer = cudaSuccess;
  g_launches.clear();
  CHECK(one_step(1000) == SAMPO_OK);
  CHECK(g_launches["small"] == 1 && g_launches["count"] == 0);
}

// The array keeps what the calls before left in it - also of two that were
// made at once, which the header rules out but cannot prevent: a one-launch
// hour starts from zero rows all the same.
static void every_call_starts_from_zero_rows() {
  memset(((Scratch*)g_fake_symbol)->small, 0x11, sizeof(Scratch::small));
  g_launches.clear();
  CHECK(one_step(1000) == SAMPO_OK);
  CHECK(g_launches["small"] == 1 && g_launches["small on clean rows"] == 1);
}

int main() {
  every_call_starts_from_zero_rows();
  refused_launches_take_the_passes();
  printf(g_checks_failed ? "%d checks failed\n" : "ok\n", g_checks_failed);
  return g_checks_failed ? 1 : 0;
}
