// sampo_kernels.cuh - device state shared by the kernels and the host API.
//
// The kernels step a batch of independent simulations ("replicates") at
// once: every replicate has its own pool buffers, state, span arrays and
// input rings (RepParams), and the persistent kernels' warps take the spans of
// all active replicates in turn. A single simulation is a batch of one.
#pragma once
#include <stdint.h>
#ifndef __CUDACC_RTC__
#include <string.h>
#include <algorithm>
#endif
#include "../../include/sampo.h"
#include "sampo_math.h"
#include "sampo_model.cuh"

namespace sampo {

constexpr int kBlock = 256;                 // threads per CTA
constexpr int kItems = 4;                   // rows of 32 slots a warp of the count and update/scatter passes loads at once (2 or 4)
constexpr int kTile = kBlock * 4;           // slots per tile of the one-launch step at its largest
constexpr int kWarps = kBlock / 32;
constexpr uint32_t kMaxRep = 1024;          // replicates per batch

// One pool buffer: structure of arrays, one column per agent field.
struct DevPool {
  float* age; float* his; float* delay; float* sporo;
  uint32_t* uni; uint32_t* avail; uint32_t* cycle; uint32_t* hbc; uint32_t* batches;
  uint8_t* flags;   // bits 0-2 state (0..7), bit 3 isFemale
};

// Device-resident state of one simulation.
// A glibc rand() stream held on the device (generateSeeds, src/abms.c:145-150,
// drawn by k_publish for each coming step). The 31 words are kept rotated so
// that st.r[0] is the oldest (the next draw is r[0] + r[28]); st.i is a
// multiple of 31, so the state also continues on the host's sampo_rand_next.
struct DevSeedStream {
  uint32_t next;              // step whose seeds are drawn next; kNoStream: seeds come from the host
  sampo_rand_state st;
};
constexpr uint32_t kNoStream = 0xffffffffu;

// What the decisions of one step add up to, besides the survivor counts.
struct Decided {
  uint32_t newEggs;           // eggs laid (EggsNbiomass.newEggs)
  uint32_t L1de, dmin, dmax;  // the larvae of the pool it makes: L1de, youngest and oldest age in days
};

struct SimDev {
  sampo_population pop;       // ranges + stats of the current pool (reference pop[0] at step start)
  sampo_bites_cycles bnc;     // counters of the last update (printed with the next row)
  sampo_stats_row begun;      // the row of the step that k_begin_step began
  uint32_t step;              // index of the next step
  uint32_t cur;               // current pool buffer (0/1)
  // The decided step: what its decisions (count pass, or the update/scatter
  // pass of the step before) make of the pool.
  Decided dec;
  uint32_t cnt[8];            // its survivors by next state
  Decided ahead_dec;          // the same of the step after, while a pass decides ahead
  uint32_t ahead;             // the running step's update/scatter pass decides the step after
  uint32_t rot;               // the span counts of the decided step: RepParams::spans + rot * spanStride
  uint32_t dirty[3];          // spans of each of the three that may not be zero
  uint32_t spans_done;        // count pass: spans counted so far
  uint32_t acc_bnc[4];        // update/scatter pass: numCycles, sumCycles, numBites, numInfectBites
  uint32_t acc_fem, acc_inf;  // females and potentially infective ones of the next pool
  uint32_t error;             // sticky SAMPO_DEV_ERR_* bits
  uint32_t warn;              // sticky SAMPO_DEV_WARN_* bits
  uint32_t capacity;
  float cc;                   // carrying capacity (constant per run, src/abms.c:19,132)
  uint32_t active;            // 1: the replicate takes part in the batch's steps
  uint32_t stop_step;         // becomes inactive once step reaches this
  uint32_t wide;              // k_pool_stats: the pool holds a record its state does not imply (state_cols)
  DevSeedStream rnd;          // the replicate's own rand() stream, when its seeds are drawn on the device
  StepCtx ctx[2];             // constants of step s at s % 2 (the coming step's valid while active)
  uint32_t larvaKill[2][100]; // larval mortality of step s by age in days (kill_threshold), at s % 2
};

// Batch-wide state.
struct BatchDev {
  uint32_t minSpan;           // smallest span (slots), see span_size; set by the host between runs
  uint32_t bar;               // one-launch step: CTAs past the decision phase (reset by its last CTA)
  uint32_t done;              // one-launch step: CTAs finished (reset by its last CTA)
};

__host__ __device__ constexpr uint32_t units_of(uint32_t n, uint32_t size) { return n / size + (n % size ? 1u : 0u); }

// The inputs of one step.
struct CtxInputs {
  sampo_seeds sd[4];
  sampo_environment env;
  float T;
  uint32_t wt;
};

// The one-launch step's rows for pools of up to `tiles` 256-slot tiles
// (sampo_small_step.cuh): three sets of group records, a 16-byte word per
// tile, four words of state. The records and the state start from zero.
constexpr uint32_t kSmallGroupTiles = 16, kSmallGroupWords = 16;
__host__ __device__ constexpr size_t small_group_words(uint32_t tiles) {
  return 3 * (size_t)units_of(tiles, kSmallGroupTiles) * kSmallGroupWords;
}
__host__ __device__ constexpr size_t small_row_words(uint32_t tiles) { return small_group_words(tiles) + 4 * (size_t)tiles + 4; }

// Spans: the slots a warp of the two passes takes at once, a multiple of 32.
// A span costs a warp about a thousand instructions besides its rows (its
// prefix, the start and end of its range, the agents that move on in a
// partly filled warp), a row of 32 agents 60 to 150, so a pool is cut into as
// few spans as keep every warp of the resident grid equally busy: the smallest
// multiple of kSpanWarps that keeps them at kSpanMax slots. kSpanWarps is the
// resident grid of a GB300, 152 SMs x 3 CTAs (what the passes' 80 registers
// and 59 KB of shared memory allow) x 8 warps; a constant, because the spans
// are sized where no host call can ask (the kernels and the sizes of the span
// arrays). A grid of fewer warps takes the spans in more turns, to the same
// results. A batch sets a larger smallest span (BatchDev::minSpan), since its
// replicates share the warps.
constexpr uint32_t kSpanMin = 128, kSpanMax = 1024, kSpanWarps = 152 * 3 * 8;
__host__ __device__ constexpr uint32_t span_size(uint32_t end, uint32_t min_span) {
  const uint32_t warps = kSpanWarps * (end / (kSpanWarps * kSpanMax) + 1u);
  uint32_t s = units_of(end, warps);
  s = s < kSpanMin ? kSpanMin : s;
  s = s < min_span ? min_span : s;
  s = (s + 31u) / 32u * 32u;
  return s < kSpanMax ? s : kSpanMax;
}
__host__ __device__ constexpr uint32_t span_count(uint32_t end, uint32_t min_span) { return units_of(end, span_size(end, min_span)); }
// The most spans any pool of up to `capacity` slots has.
__host__ __device__ constexpr uint32_t max_spans(uint32_t capacity) {
  const uint32_t a = capacity / kSpanMin + 1u, b = capacity / kSpanMax + kSpanWarps + 1u;
  return a < b ? a : b;
}
// The span arrays of a pool of `capacity` slots, in 16-byte words: a span's
// survivors by next state (one word, for each of three steps), a super's (32
// spans) the same, and its exclusive prefix (two).
__host__ __device__ constexpr uint32_t max_supers(uint32_t capacity) { return (max_spans(capacity) + 31u) / 32u; }
__host__ __device__ constexpr size_t span_array_words(uint32_t capacity) {
  return 3 * ((size_t)max_spans(capacity) + max_supers(capacity));
}

// Everything the kernels need of one replicate.
struct RepParams {
  SimDev* sim;
  DevPool pool[2];
  uint8_t* dec;               // caller-owned pools: [slots] the count pass's decisions; null: they are in the flags
  uint4* spans;               // [3][spanStride] survivors by next state, 16 bits each: of the decided step, of the step
                              // after (while deciding ahead), and the one cleared for the step after that
  uint4* supers;              // [max_supers] the same of 32 spans, while they are being counted; zero otherwise
  uint32_t* superPre;         // [max_supers][8] survivors of the supers before, of the decided step
  uint32_t spanStride;
  uint32_t* smallRows;        // one-launch step: small_row_words(smallTiles) words (16-byte aligned), or null
  uint32_t smallTiles;
  float* T;                   // [ring] temperature per step
  sampo_environment* env;     // [ring]
  sampo_seeds* seeds;         // [ring][4] (written by the device for a device seed stream)
  uint32_t* wt;               // [ring] world time per step
  sampo_stats_row* rows;      // [ring] stats at the start of each step
  uint32_t ring;
};

struct KParams {
  const RepParams* reps;      // device array [nrep]
  uint32_t nrep;
  BatchDev* bat;
  const ModelConst* mc;
  const void* ks;             // host: the kernels compiled for a user species (sampo_species.cu), or null
  uint32_t wide;              // the pools hold whole records (state_cols)
};

// Modes of k_publish: PUB_AFTER_STEP turns the step's counts into the next
// pool's start; PUB_INITIAL publishes the current pool (after init/load);
// PUB_REFRESH recomputes the coming step's input-dependent constants (run it
// after writing that step's inputs); PUB_DECIDED follows a count pass whose
// update/scatter pass decides ahead. PUB_DECIDED and PUB_AFTER_STEP take
// PUB_AHEAD when the update/scatter pass that comes next decides ahead.
// Flags of k_pool_stats.
enum : uint32_t { PS_CHECK = 1, PS_CLEAR = 2, PS_ROWS = 4 };
enum : int { PUB_INITIAL = 0, PUB_AFTER_STEP = 1, PUB_REFRESH = 2, PUB_DECIDED = 3, PUB_MODE = 3, PUB_AHEAD = 4 };

#ifndef __CUDACC_RTC__  // host side (the run-time compiler sees the device part only)

// Hourly mortality tables that do not change during a run
// (kernel/killAgents.cl:84-115,135-147), computed on the host with the same
// deterministic functions the device uses.
inline void fill_constant_tables(ModelConst& h) {
  for (int d = 0; d < 100; d++) {
    const float a = 0.1f, B = 25.0f, sg = 0.1f;
    float e = sampo_expf((float)(uint32_t)d / B);
    float dmr = (a * e) / (1.0f + (a * B * sg * (e - 1.0f)));
    float dsr = 1.0f - dmr;
    float hsr = sampo_powf(dsr, 1.0f / 24.0f);
    h.kill.adult[d] = kill_threshold(1.0f - hsr);
  }
  float dmr = 0.1f;
  float dsr = 1.0f - dmr;
  h.kill.aquatic = kill_threshold(1.0f - sampo_powf(dsr, 1.0f / 24.0f));
  for (uint32_t k = 0; k < kEggBatchTable; k++) h.eggBatchScale[k] = egg_batch_scale(k);
}

// The span arrays of a pool of `capacity` slots at base (16-byte aligned,
// span_array_words words; they start as zeros).
inline void set_span_arrays(RepParams& r, void* base, uint32_t capacity) {
  r.supers = reinterpret_cast<uint4*>(base);
  r.superPre = reinterpret_cast<uint32_t*>(r.supers + max_supers(capacity));
  r.spans = r.supers + 3 * (size_t)max_supers(capacity);
  r.spanStride = max_spans(capacity);
}
inline size_t span_array_bytes(uint32_t capacity) { return span_array_words(capacity) * sizeof(uint4); }

// Why a pool's ranges cannot be stepped, or null when they can: the egg
// range starts at slot 0, no range ends before it starts, the ranges are
// ordered with a gap between them (every layout kernel/oldToNewAgents.cl:57-95
// and createInitialPopulation, src/abms.c:185-228, produce), and the pool's
// end fits `capacity`. Shared by every entry point that takes ranges from
// its caller or from a file.
inline const char* ranges_error(const sampo_population& pop, uint64_t capacity) {
  if (pop.r[0].start != 0) return "the egg range must start at slot 0";
  for (int k = 0; k < 8; k++) {
    if (pop.r[k].end < pop.r[k].start) return "range end before start";
    if (k > 0 && pop.r[k].start <= pop.r[k - 1].end) return "ranges must be ordered with a gap";
  }
  if ((uint64_t)pop.r[7].end > capacity) return "pool exceeds the capacity";
  return nullptr;
}

// Initial device state of a simulation (before its pool is published).
inline SimDev initial_sim_state(uint32_t capacity, float cc) {
  SimDev h;
  memset(&h, 0, sizeof(h));
  h.capacity = capacity;
  h.cc = cc;
  h.dec.dmin = 0xffffffffu;
  h.ahead_dec.dmin = 0xffffffffu;
  h.stop_step = 0xffffffffu;
  h.rnd.next = kNoStream;
  return h;
}

// Launch helpers (sampo_kernels.cu). The step kernels take every replicate of
// p; init, pool statistics and the histogram take p.reps[0] only. They launch
// the built-in kernels, or p.ks's when a species was compiled at run time.
// persistent grid sizes (CTAs resident on all SMs) for batches of nrep replicates
int grid_blocks_count(uint32_t nrep, const void* ks = nullptr, int items = kItems, bool wide = false);
int grid_blocks_scatter(uint32_t nrep, const void* ks = nullptr, int items = kItems, bool wide = false);
// The current device's SMs.
int device_sms();
// The grids that sampo_set_grids or the tuner chose, in CTAs per SM of the
// count and update/scatter passes; 0: the largest. They hold for every pool
// the passes run on, as far as the grid of its kernels reaches.
// (Choices of up to kCountGrids CTAs of the count pass are taken: five were
// resident before it kept a ring of chunks per warp, three are now.)
constexpr int kCountGrids = 5;
struct ChosenGrids {
  uint32_t count = 0, scatter = 0;
};
inline int chosen_grid(uint32_t chosen, int largest) { return chosen ? std::min((int)chosen * device_sms(), largest) : largest; }
// The kernels of a run-time species (sampo_species.cu): launch one, and its
// resident CTAs per SM.
enum : int {
  KID_COUNT, KID_SCATTER, KID_COUNT_WIDE, KID_SCATTER_WIDE, KID_PUBLISH, KID_INIT_EGGS, KID_POOL_STATS, KID_HISTOGRAM,
  KID_TRIAL_RESET, KID_WIDEN, KID_SMALL1, KID_SMALL2, KID_SMALL4, KID_BEGIN_STEP, KID_N
};
cudaError_t species_launch(const void* ks, int kid, dim3 grid, dim3 block, size_t smem, cudaStream_t st, void** args,
                           bool cooperative = false);
int species_occupancy(const void* ks, int kid, int threads, size_t smem);
// dynamic shared memory the two passes may request
size_t pass_smem_max();
// (the built-in passes for `items` = 2 or 4 rows at once; a run-time species
// is built for 4; p.wide picks the passes that move whole records)
cudaError_t launch_count(const KParams& p, int grid, cudaStream_t st, int items = kItems);
cudaError_t launch_scatter(const KParams& p, int grid, cudaStream_t st, int items = kItems, bool ahead = false);
// Whether the passes decide ahead over several hours (launch_steps): the
// built-in species on narrow pools.
inline bool can_decide_ahead(const KParams& p) { return !p.ks && !p.wide; }
// `nsteps` hourly steps of every replicate of p. Deciding ahead: one count
// pass, then an update/scatter pass and a publish per hour; otherwise the
// three kernels every hour.
cudaError_t launch_steps(const KParams& p, uint32_t nsteps, bool ahead, int grid_count, int grid_scatter, int items, cudaStream_t st,
                         uint32_t* launches);
// k_publish over every replicate of p (modes PUB_*, above).
cudaError_t launch_publish(const KParams& p, int mode, cudaStream_t st);
// (`full`: every column, else those that hold an egg's record in a narrow pool)
cudaError_t launch_init_eggs(const KParams& p, uint32_t n, float T0, const sampo_seeds* seeds_dev,
                             int age_days_max, uint64_t age_seed, bool full, cudaStream_t st);
// statistics of p.reps[0]'s current pool, then its publish (PUB_INITIAL);
// `check` also finds out whether the pool is a wide one (SimDev::wide)
// (flags: PS_*; end: the pool's end, which sizes the grid)
cudaError_t launch_publish_start(const KParams& p, uint32_t flags, uint32_t end, cudaStream_t st);
// The coming step's inputs into ring slot `slot`, and its constants.
cudaError_t launch_begin_step(const KParams& p, const CtxInputs& in, uint32_t slot, cudaStream_t st);
// the columns that the records of p's narrow pools imply, written out, and
// the decisions taken out of the flags (before a pool is read back)
cudaError_t launch_widen(const KParams& p, cudaStream_t st);
cudaError_t launch_histogram(const KParams& p, uint32_t* hist_dev, cudaStream_t st);
// {step, active, status bits, pool end} of each of n states (n >= 1).
cudaError_t launch_slot_states(const SimDev* sims, uint32_t n, uint4* out, cudaStream_t st);
cudaError_t launch_eval_math(int fn, const float* x, const float* y, float* out, uint32_t n, cudaStream_t st);
// Kernel nodes in a captured graph (the launches one replay makes).
cudaError_t graph_kernel_nodes(cudaGraph_t g, uint32_t* kernels);
// The one-launch steps of a single simulation (sampo_small_step.cuh) with
// tiles of kBlock * items slots (items 1, 2 or 4), built in or of ks: the
// largest grid (CTAs resident on all SMs, 0 if it cannot run) and a launch of `nsteps` hourly
// steps (a cooperative launch when `cooperative`) on `grid` CTAs.
int grid_blocks_small(int items = kItems, const void* ks = nullptr);
// The largest grid all three tile sizes can take.
int grid_blocks_small_all(const void* ks);
// A step or day on a pool that ends at `end`: the smallest tiles (the shortest
// chain of updates per thread) of which `growth` times the pool's fit `grid`
// CTAs, as slots per thread.
inline int small_items_for(uint32_t end, uint32_t growth, int grid) {
  for (int i : {1, 2})
    if ((uint64_t)std::max(units_of(end, (uint32_t)(kBlock * i)), 1u) * growth <= (uint64_t)grid) return i;
  return 4;
}
// One hour now: every tile its CTA and one more, which prepares the next hour.
cudaError_t launch_small_hour(const KParams& p, uint32_t end, int items, int max_grid, cudaStream_t st);
cudaError_t launch_small(const KParams& p, int grid, bool cooperative, uint32_t nsteps, cudaStream_t st,
                         int items = kItems);
// Times count + scatter of the coming step for each number of rows at once
// (4 and, for the built-in species, 2) at every (count, scatter) number of
// CTAs per SM the occupancy allows, and returns the fastest. The scatter pass
// timed is the one that does not decide ahead (single hours, whole records,
// run-time species, small batches); days that decide ahead run it one hour in
// 24 and k_count once, and take its picks over. The trials leave the
// simulations' course unchanged (k_trial_reset); the coming step's constants
// must be current (PUB_REFRESH) before the call.
cudaError_t tune_grids(const KParams& p, cudaStream_t st, int* grid_count, int* grid_scatter, int* items, double* best_ms);

#endif  // __CUDACC_RTC__

}  // namespace sampo
