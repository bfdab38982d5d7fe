/*
 * host_batch_check.cu - the host side of the batches (sampo_batch.cu) on
 * fake_cuda.h: what a call leaves in a slot's device state.
 */
#include "fake_cuda.h"
#include "../sampo_gb300/csrc/sampo_batch.cu"

// A batch of one slot with a population, its ring filled with inputs.
static sampo_batch* one_slot(uint64_t capacity, uint32_t* slot) {
  sampo_batch* b = nullptr;
  sampo_batch_config bc = {2, 16, 0};
  CHECK(sampo_batch_create(&bc, &b) == SAMPO_OK);
  sampo_replicate_config rc = {capacity, 1000.0f, 0xffffffffu};
  CHECK(sampo_batch_add(b, &rc, slot) == SAMPO_OK);
  float T[16];
  sampo_environment env[16];
  memset(env, 0, sizeof(env));
  for (int i = 0; i < 16; i++) {
    T[i] = 20.0f + (float)i;
    env[i].carryingCapacity = 1000.0f;
  }
  CHECK(sampo_batch_set_inputs(b, *slot, 0, T, env, 16) == SAMPO_OK);
  sampo_seeds seeds[4];
  memset(seeds, 0, sizeof(seeds));
  CHECK(sampo_batch_init_population(b, *slot, 100, seeds, 0, 0) == SAMPO_OK);
  return b;
}

// The update/scatter pass that decides ahead clears dirty[rot - 1] words of
// the span counts before the decided ones and adds to those after them, which
// must be zero: whatever a slot brings into a (smaller) allocation, the counts
// it says are to be cleared lie inside the new arrays and the new arrays are
// all zero.
static void grown_slots_have_clean_span_counts() {
  for (uint32_t rot = 0; rot < 3; rot++) {
    uint32_t slot = 0;
    sampo_batch* b = one_slot(1u << 20, &slot);
    SimDev* sim = b->sims_dev + slot;
    sim->rot = rot;
    for (uint32_t k = 0; k < 3; k++) sim->dirty[k] = max_spans(1u << 20) - k;
    sim->spans_done = 3;
    CHECK(sampo_batch_grow(b, slot, 1024) == SAMPO_OK);
    const RepParams& rp = b->reps_dev[slot];
    CHECK(rp.spanStride == max_spans(1024));
    CHECK(sim->rot < 3);
    for (uint32_t k = 0; k < 3; k++) CHECK(sim->dirty[k] == 0);
    CHECK(sim->spans_done == 0);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(rp.supers);
    bool zero = true;
    for (size_t i = 0; i < span_array_bytes(1024) / 4; i++) zero &= w[i] == 0;
    CHECK(zero);
    for (int i = 0; i < 16; i++) CHECK(rp.T[i] == 20.0f + (float)i);
    CHECK(sampo_batch_destroy(b) == SAMPO_OK);
  }
}

// Resumes a slot from a checkpoint whose records are, or are not, implied by
// their states.
static void resume(sampo_batch* b, uint32_t slot, const char* path, bool wide) {
  g_wide_found = wide;
  CHECK(sampo_batch_checkpoint_load(b, slot, path) == SAMPO_OK);
}
static bool grids_are(const sampo_batch* b, int count, int scatter) {
  return b->grid_count == count * kFakeSms && b->grid_scatter == scatter * kFakeSms;
}

// Chosen grids stay chosen when a slot's pool makes the batch move whole records.
static void chosen_grids_outlive_a_wide_pool() {
  const char* path = "sampo_fake_batch.ck";
  for (bool tuned : {false, true}) {
    uint32_t slot = 0;
    sampo_batch* b = one_slot(4096, &slot);
    CHECK(sampo_batch_checkpoint_save(b, slot, path) == SAMPO_OK);
    CHECK(grids_are(b, 3, 3));
    if (tuned) {
      b->reps[slot].seed_step[0] = 0;
      CHECK(sampo_batch_autotune(b, nullptr, nullptr) == SAMPO_OK);
    } else {
      CHECK(sampo_batch_set_grids(b, 2, 1) == SAMPO_OK);
    }
    resume(b, slot, path, true);
    CHECK(b->wide);
    CHECK(grids_are(b, 2, 1));
    CHECK(sampo_batch_set_items_per_thread(b, 2) == SAMPO_OK);
    CHECK(grids_are(b, 3, 3));
    CHECK(sampo_batch_destroy(b) == SAMPO_OK);
  }
  remove(path);
}

static void choices_of_smaller_kernels_are_taken() {
  uint32_t slot = 0;
  sampo_batch* b = one_slot(4096, &slot);
  CHECK(sampo_batch_set_grids(b, 5, 2) == SAMPO_OK && grids_are(b, 3, 2));
  CHECK(sampo_batch_set_grids(b, 6, 2) == SAMPO_ERR_ARG);
  CHECK(sampo_batch_destroy(b) == SAMPO_OK);
}

// A batch moves whole records while a slot of it holds a pool that needs
// them, and no longer: removing the slot, or putting another population into
// it, ends it; the other slots' pools get their implied columns at its start.
static void whole_records_only_while_a_slot_needs_them() {
  const char* path = "sampo_fake_batch.ck";
  for (int end : {0, 1, 2}) {
    uint32_t slot = 0, other = 0;
    sampo_batch* b = one_slot(4096, &slot);
    CHECK(sampo_batch_checkpoint_save(b, slot, path) == SAMPO_OK);
    const sampo_replicate_config rc = {4096, 1000.0f, 0xffffffffu};
    CHECK(sampo_batch_add(b, &rc, &other) == SAMPO_OK && other != slot);
    g_launches.clear();
    resume(b, other, path, true);
    CHECK(b->wide && g_launches["widen"] == 1);
    if (end == 0) {
      CHECK(sampo_batch_remove(b, other) == SAMPO_OK);
    } else if (end == 1) {
      resume(b, other, path, false);
    } else {
      sampo_seeds seeds[4];
      memset(seeds, 0, sizeof(seeds));
      b->reps[other].input_step[0] = 0;
      CHECK(sampo_batch_init_population(b, other, 100, seeds, 0, 0) == SAMPO_OK);
      CHECK(g_launches["init, whole"] == 0);
    }
    CHECK(!b->wide);
    resume(b, slot, path, true);
    CHECK(b->wide);
    resume(b, slot, path, true);
    CHECK(b->wide);
    CHECK(sampo_batch_destroy(b) == SAMPO_OK);
  }
  remove(path);
}

int main() {
  whole_records_only_while_a_slot_needs_them();
  choices_of_smaller_kernels_are_taken();
  chosen_grids_outlive_a_wide_pool();
  grown_slots_have_clean_span_counts();
  printf(g_checks_failed ? "%d checks failed\n" : "ok\n", g_checks_failed);
  return g_checks_failed ? 1 : 0;
}
