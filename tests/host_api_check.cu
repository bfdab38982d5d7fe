/*
 * host_api_check.cu - the host side of a single simulation (sampo_api.cu) on
 * fake_cuda.h.
 */
#include "fake_cuda.h"
#include "../sampo_gb300/csrc/sampo_api.cu"

// A simulation with inputs and a population of 100 eggs.
static sampo_sim* with_pool() {
  sampo_sim* s = nullptr;
  const sampo_config cfg = {4096, 1000.0f, 0, 16};
  CHECK(sampo_create(&cfg, &s) == SAMPO_OK);
  float T[16];
  sampo_environment env[16];
  sampo_seeds seeds[64];
  memset(env, 0, sizeof(env));
  memset(seeds, 0, sizeof(seeds));
  for (int i = 0; i < 16; i++) {
    T[i] = 25.0f;
    env[i].carryingCapacity = 1000.0f;
  }
  CHECK(sampo_set_inputs(s, 0, T, env, 16) == SAMPO_OK);
  CHECK(sampo_set_seeds(s, 0, seeds, 16) == SAMPO_OK);
  CHECK(sampo_init_population(s, 100, seeds, 0, 0) == SAMPO_OK);
  return s;
}
static int one_step(sampo_sim* s) {
  sampo_environment env;
  memset(&env, 0, sizeof(env));
  env.carryingCapacity = 1000.0f;
  sampo_seeds seeds[4];
  memset(seeds, 0, sizeof(seeds));
  sampo_stats_row row;
  return sampo_step(s, &env, 25.0f, 0, seeds, &row);
}

// A one-launch hour that gave up (here: the bits such a launch sets, and
// counts left in its records) leaves records that the next one adds to: they
// are zero again before the next one-launch hour, whichever call comes first
// and whether the bits have been read and cleared since.
static void records_are_zero_after_a_launch_that_gave_up() {
  for (uint32_t bit : {(uint32_t)SAMPO_DEV_ERR_BARRIER, (uint32_t)SAMPO_DEV_ERR_TMA})
    for (int clear_by : {0, 1, 2})
      for (int go_on : {0, 1, 2}) {
        sampo_sim* s = with_pool();
        const char* path = "sampo_fake.ck";
        CHECK(sampo_checkpoint_save(s, path) == SAMPO_OK);
        CHECK(one_step(s) == SAMPO_OK);
        const size_t words = small_row_words(units_of(4096, 256));
        memset(s->small_mem, 0x11, words * 4);
        s->bat_dev->bar = s->bat_dev->done = 7;
        s->sim_dev->error = bit;
        if (clear_by != 2) CHECK(one_step(s) == SAMPO_ERR_INTERNAL);
        uint32_t bits = 0;
        if (clear_by) {
          CHECK(sampo_device_status(s, &bits, 1) == SAMPO_OK && bits == bit);
          // hours of the three kernels meanwhile: the status words read last are clean
          CHECK(sampo_set_small_step(s, 0) == SAMPO_OK);
          CHECK(one_step(s) == SAMPO_OK);
          CHECK(sampo_set_small_step(s, SAMPO_SMALL_STEP_DEFAULT) == SAMPO_OK);
        }
        if (go_on == 1) CHECK(sampo_checkpoint_load(s, path) == SAMPO_OK);
        if (go_on == 2) {
          sampo_seeds seeds[4];
          memset(seeds, 0, sizeof(seeds));
          CHECK(sampo_init_population(s, 100, seeds, 0, 0) == SAMPO_OK);
        }
        g_launches.clear();
        (void)one_step(s);
        CHECK(g_launches["small"] == 1 && g_launches["small on clean rows"] == 1);
        CHECK(sampo_destroy(s) == SAMPO_OK);
        remove(path);
      }
}

// Where the device refuses the cooperative launch (a stream that owns part of
// the SMs, say), the hour is stepped by the three kernels.
static void refused_launches_take_the_three_kernels() {
  sampo_sim* s = with_pool();
  g_small_answer = cudaErrorCooperativeLaunchTooLarge;
  g_launches.clear();
  const uint64_t before = s->launches;
  CHECK(one_step(s) == SAMPO_OK);
  CHECK(g_launches["begin"] == 1 && g_launches["small"] == 1 && g_launches["steps"] == 1);
  CHECK(s->launches - before == 4);  // (the refused one did not run)
  g_small_answer = cudaSuccess;
  g_launches.clear();
  CHECK(one_step(s) == SAMPO_OK);
  CHECK(g_launches["small"] == 1 && g_launches["steps"] == 0);
  CHECK(sampo_destroy(s) == SAMPO_OK);
}

// Puts a pool in place whose records are, or are not, implied by their states.
static void load_pool(sampo_sim* s, bool wide) {
  uint32_t words[128];
  uint8_t bytes[128];
  memset(words, 0, sizeof(words));
  memset(bytes, 0, sizeof(bytes));
  sampo_population pop;
  memset(&pop, 0, sizeof(pop));
  pop.r[0].end = 16;
  for (uint32_t k = 1; k < 8; k++) pop.r[k].start = pop.r[k].end = 16 + k;
  sampo_pool_view v = {(float*)words, (float*)words, (float*)words, (float*)words, words, words, words, words, words, bytes, bytes};
  g_wide_found = wide;
  CHECK(sampo_load_pool(s, &pop, &v) == SAMPO_OK);
  CHECK(s->wide == wide);
}
static bool grids_are(const sampo_sim* s, int count, int scatter) {
  return s->grid_count == count * kFakeSms && s->grid_scatter == scatter * kFakeSms;
}

// Grids that the caller or the tuner chose stay chosen when a pool of the
// other kind of records is loaded, as far as its passes reach; the calls that
// reset them to the largest (the number of rows at once, the species) do.
static void chosen_grids_outlive_the_pool() {
  for (bool tuned : {false, true}) {
    sampo_sim* s = with_pool();
    g_resident = 3;
    g_resident_wide = 3;
    CHECK(grids_are(s, 3, 3));
    load_pool(s, true);
    CHECK(grids_are(s, 3, 3));
    g_resident_wide = 2;  // (as the largest grids of the passes differ)
    load_pool(s, false);
    load_pool(s, true);
    CHECK(grids_are(s, 2, 2));
    load_pool(s, false);
    if (tuned) {  // picks (2, 1)
      CHECK(sampo_autotune(s, nullptr, nullptr) == SAMPO_OK);
    } else {
      CHECK(sampo_set_grids(s, 2, 1) == SAMPO_OK);
    }
    CHECK(grids_are(s, 2, 1));
    load_pool(s, true);
    CHECK(grids_are(s, 2, 1));
    load_pool(s, false);
    CHECK(grids_are(s, 2, 1));
    g_resident_wide = 1;
    load_pool(s, true);
    CHECK(grids_are(s, 1, 1));
    load_pool(s, false);
    CHECK(grids_are(s, 2, 1));
    CHECK(sampo_set_items_per_thread(s, 2) == SAMPO_OK);
    CHECK(grids_are(s, 3, 3));
    CHECK(sampo_destroy(s) == SAMPO_OK);
  }
}

// What an earlier build's tuner chose, with up to 5 CTAs of the count pass on
// an SM, is still taken, and runs as the largest grid.
static void choices_of_smaller_kernels_are_taken() {
  sampo_sim* s = with_pool();
  g_resident = 3;
  for (uint32_t c = 1; c <= 5; c++) {
    CHECK(sampo_set_grids(s, c, 2) == SAMPO_OK);
    CHECK(grids_are(s, (int)std::min(c, 3u), 2));
  }
  CHECK(sampo_set_grids(s, 6, 2) == SAMPO_ERR_ARG);
  CHECK(sampo_set_grids(s, 1, 4) == SAMPO_ERR_ARG);
  CHECK(sampo_set_grids(s, 0, 1) == SAMPO_ERR_ARG);
  CHECK(grids_are(s, 3, 2));
  CHECK(sampo_destroy(s) == SAMPO_OK);
}

int main() {
  choices_of_smaller_kernels_are_taken();
  chosen_grids_outlive_the_pool();
  refused_launches_take_the_three_kernels();
  records_are_zero_after_a_launch_that_gave_up();
  printf(g_checks_failed ? "%d checks failed\n" : "ok\n", g_checks_failed);
  return g_checks_failed ? 1 : 0;
}
