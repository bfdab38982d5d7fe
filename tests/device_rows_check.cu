/*
 * device_rows_check.cu - days of one-launch steps behind one that gave up
 * waiting: here the mark that such a launch leaves in its rows, and counts
 * left in its records, put there by the host. The queued days do nothing and
 * report it, and the simulation goes on from its checkpoint as if nothing
 * had been. Built with the library's objects (its kernels), on a GPU.
 */
#include "../sampo_gb300/csrc/sampo_api.cu"

#define CHECK(x)                                     \
  do {                                               \
    if (!(x)) {                                      \
      printf("%s:%d: %s\n", __FILE__, __LINE__, #x); \
      return 1;                                      \
    }                                                \
  } while (0)

static const int kHours = 96;

static sampo_sim* start() {
  sampo_sim* s = nullptr;
  const sampo_config cfg = {1 << 16, 20000.0f, 0, kHours + 1};
  if (sampo_create(&cfg, &s) != SAMPO_OK) return nullptr;
  std::vector<float> T(kHours, 27.0f);
  std::vector<sampo_environment> env(kHours);
  std::vector<sampo_seeds> seeds(4 * (kHours + 1));
  for (auto& e : env) {
    memset(&e, 0, sizeof(e));
    e.bloodmealSuccess = 0.25f;
    e.carryingCapacity = 20000.0f;
  }
  uint32_t* w = reinterpret_cast<uint32_t*>(seeds.data());
  for (size_t i = 0; i < seeds.size() * 4; i++) w[i] = 1000u + (uint32_t)i * 2654435761u % 1000000007u;
  if (sampo_set_inputs(s, 0, T.data(), env.data(), kHours) != SAMPO_OK || sampo_set_seeds(s, 0, seeds.data(), kHours) != SAMPO_OK ||
      sampo_init_population(s, 8000, seeds.data() + 4 * kHours, 3, 5) != SAMPO_OK)
    return nullptr;
  return s;
}

int main(int argc, char** argv) {
  CHECK(argc == 2);
  std::vector<sampo_stats_row> want(kHours), got(kHours);
  sampo_sim* s = start();
  CHECK(s && sampo_run(s, kHours, want.data()) == SAMPO_OK && s->days_small == kHours / 24);
  CHECK(sampo_destroy(s) == SAMPO_OK);

  s = start();
  CHECK(s && sampo_run(s, 24, got.data()) == SAMPO_OK && sampo_checkpoint_save(s, argv[1]) == SAMPO_OK);
  SimDev before, after;
  CHECK(cudaMemcpy(&before, s->sim_dev, sizeof(before), cudaMemcpyDeviceToHost) == cudaSuccess);
  const uint32_t tiles = units_of(1 << 16, 256);
  const size_t groups = small_group_words(tiles), words = small_row_words(tiles);
  std::vector<uint32_t> left(words, 0u);
  for (size_t i = 0; i < groups; i++) left[i] = 0x00010001u;
  left[words - 1] = 1u;
  CHECK(cudaMemcpy(s->small_mem, left.data(), words * 4, cudaMemcpyHostToDevice) == cudaSuccess);
  CHECK(sampo_run(s, 48, got.data() + 24) == SAMPO_ERR_INTERNAL);
  CHECK(cudaMemcpy(&after, s->sim_dev, sizeof(after), cudaMemcpyDeviceToHost) == cudaSuccess);
  CHECK(after.error == SAMPO_DEV_ERR_BARRIER && after.step == before.step && after.cur == before.cur);
  CHECK(memcmp(&after.pop, &before.pop, sizeof(after.pop)) == 0);
  uint32_t bits = 0;
  CHECK(sampo_device_status(s, &bits, 1) == SAMPO_OK && bits == SAMPO_DEV_ERR_BARRIER);
  CHECK(sampo_checkpoint_load(s, argv[1]) == SAMPO_OK);
  CHECK(sampo_run(s, kHours - 24, got.data() + 24) == SAMPO_OK);
  CHECK(memcmp(got.data(), want.data(), kHours * sizeof(sampo_stats_row)) == 0);
  CHECK(s->days_small >= 2 && sampo_destroy(s) == SAMPO_OK);
  printf("ok\n");
  return 0;
}
