// sampo_step_kernels.cuh - the device code of the SAMPO hourly step (sm_103a):
// helpers, k_count, k_publish, k_scatter and the pool kernels. Compiled into
// the library by nvcc (sampo_kernels.cu) and, for a user species header, at
// run time by NVRTC (sampo_species.cu).
//
// A day of a batch of simulations is one k_count, then 24 k_scatter, each of
// which decides the hour after its own as it writes, and after each of these
// kernels a k_publish (launch_steps); a single hour, a run-time species, whole
// records and small batches take all three kernels every hour. k_count and
// k_scatter go over every active replicate's current pool buffer, k_publish
// has a CTA per replicate:
//
//  k_count   reads the columns that decide survival, the next state and the
//            eggs laid (killAgents + the decision part of updateAgents; 9 to
//            13 bytes of an agent with its flags, decide_cols), notes each
//            decision in two bits of the agent's flags, and counts the
//            survivors by next state per span of slots and the replicate's
//            new eggs.
//  k_scatter applies the decisions to the records (state_cols), obtains each
//            survivor's stable rank within its next state (the span counts
//            of k_count, then ballots), writes the updated record to its
//            slot in the other buffer (the reference's oldToNewAgents
//            layout, kernel/oldToNewAgents.cl:57-95,126-226), writes the new
//            eggs at [0, newEggs) (initAgents, kernel/initAgents.cl:26-65),
//            and accumulates the next step's statistics (calcL1de.cl,
//            calcGender.cl).
//  k_publish turns each replicate's counts into its next population, stats
//            row, step constants and larval mortality table.
//
// This replaces the reference's 19 kernels per step (killAgents,
// updateAgents, initAgents, 3 x preScan + 3 x Bolt scan-by-key,
// oldToNewAgents, calcL1de x2, calcFemales x2) and its blocking transfers.
#pragma once
#ifndef __CUDACC_RTC__
#include <stddef.h>
#endif
#include "sampo_kernels.cuh"

namespace sampo {


constexpr uint32_t kWaitLimit = 1u << 22;                    // bounded mbarrier waits

// ---------------- memory-model and TMA helpers ----------------
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// 1-D bulk copy global -> shared, completion counted on bar (both addresses
// 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Waits for the phase with the given parity; gives up after kWaitLimit polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kWaitLimit; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Range of slot g in the current layout, -1 for gaps and the tail
// (the validity test of every reference kernel, e.g. kernel/killAgents.cl:28-35).
__device__ __forceinline__ int range_of(const sampo_population& pop, uint32_t g) {
  if (g < pop.r[0].end) return 0;
#pragma unroll
  for (int k = 1; k < 8; k++) {
    if (g < pop.r[k].start) return -1;
    if (g < pop.r[k].end) return k;
  }
  return -1;
}

// Layout of the next pool from the survivor counts (kernel/oldToNewAgents.cl:57-95).
__device__ __forceinline__ void next_layout(const uint32_t cnt[8], uint32_t newEggs, sampo_population& np, uint32_t base[8]) {
  np.r[0].start = 0;
  np.r[0].end = newEggs + cnt[0];
  base[0] = newEggs;
#pragma unroll
  for (int k = 1; k < 8; k++) {
    np.r[k].start = ((np.r[k - 1].end + kLayoutAlign) / kLayoutAlign) * kLayoutAlign;
    np.r[k].end = np.r[k].start + cnt[k];
    base[k] = np.r[k].start;
  }
  np.numLarvae1DayEquiv = 0; np.numFemale = 0; np.numPotentiallyInfective = 0;
}

// Whether the next layout (kernel/oldToNewAgents.cl:57-95) fits in one buffer.
__device__ __forceinline__ bool layout_fits(const uint32_t cnt[8], uint32_t newEggs, uint32_t capacity) {
  const uint64_t tot = (uint64_t)newEggs + cnt[0];
  uint64_t e = tot;
#pragma unroll
  for (int k = 1; k < 8; k++) e = ((e + kLayoutAlign) / kLayoutAlign) * kLayoutAlign + cnt[k];
  return tot <= 0xffffffffull && e <= (uint64_t)capacity;
}

// The inputs of step `step` of one replicate (its ring slot).
__device__ __forceinline__ void load_ctx_inputs(const RepParams& rp, uint32_t step, CtxInputs& in) {
  const uint32_t i = step % rp.ring;
#pragma unroll
  for (int k = 0; k < 4; k++) in.sd[k] = rp.seeds[(size_t)i * 4 + k];
  in.env = rp.env[i];
  in.T = rp.T[i];
  in.wt = rp.wt[i];
}

// The constants of a step of one simulation starting from `pop`, from the
// step's inputs: HybridTaus with z1 and z3 folded per seed slot
// (include/gpuRand.h:33-50), the species functions of the step's temperature
// (include/properties.h) and the biomass of the pool
// (kernel/killAgents.cl:42-43). The larval mortality table is filled
// separately (k_publish).
__device__ void make_ctx(const CtxInputs& in, const uint32_t* larvaKill, const sampo_population& pop, StepCtx& c) {
  c.larvaKill = larvaKill;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    c.rng_c13[k] = taus_step(in.sd[k].z1 + 128u, 13, 19, 12, 4294967294u) ^ taus_step(in.sd[k].z3 + 128u, 3, 11, 17, 4294967280u);
    c.rng_z2[k] = in.sd[k].z2 + 128u;
    c.rng_k4[k] = 1664525u * in.sd[k].z4;
  }
  c.env = in.env;
  const float T = in.T;
  c.T = T;
  c.wt = in.wt;
  c.totalBiomass = pop.numLarvae1DayEquiv + pop.r[EGG].end + (pop.r[PUPA].end - pop.r[PUPA].start);
  species_step(T, c.wt, c);
  c.sporoOn = T > 16.0f;                                             // kernel/updateAgents.cl:69-70
  c.sporoInc = __ddiv_rn(1.0, __dmul_rn((double)(111.0f / (T - 16.0f)), 14.0));
  sampo_split_double(c.sporoInc, &c.sporoH, &c.sporoM, &c.sporoL);
}

// generateSeeds (src/abms.c:145-150) on the device: the 16 rand() draws of a
// step (z1..z4 of seed slots 0..3) from the replicate's rotated glibc TYPE_3
// state, by one warp. Lane j holds r[j]; draw k is r[k] + r[k+28] for k < 3
// and r[k] + draw(k-3) after that, resolved in five shuffle rounds. The draws
// go to the step's ring slot (output = value >> 1) and the state keeps the 31
// newest values, oldest first.
__device__ void draw_step_seeds(const RepParams& rp, uint32_t step) {
  DevSeedStream& s = rp.sim->rnd;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t x = lane < 31u ? s.st.r[lane] : 0u;
  uint32_t v = x + __shfl_sync(0xffffffffu, x, (lane + 28u) & 31u);  // final on lanes 0..2
#pragma unroll
  for (int it = 0; it < 5; it++) {  // after round it, lanes below 3 * (it + 2) are final
    const uint32_t prev = __shfl_up_sync(0xffffffffu, v, 3);
    if (lane >= 3u) v = x + prev;
  }
  uint32_t* out = reinterpret_cast<uint32_t*>(rp.seeds + (size_t)(step % rp.ring) * 4);
  if (lane < 16u) out[lane] = v >> 1;
  const uint32_t kept = __shfl_sync(0xffffffffu, x, (lane + 16u) & 31u);
  const uint32_t drawn = __shfl_sync(0xffffffffu, v, (lane + 17u) & 31u);  // lane j >= 15: draw j - 15
  if (lane < 31u) s.st.r[lane] = lane < 15u ? kept : drawn;
  if (lane == 0u) s.next = step + 1u;
}

// Puts back the last step's draws (the step's ring slot keeps them, and the
// next time they come out the same): the words from 15 on are the draws, draw
// k less the word three before it is r[k] again.
__device__ void undraw_step_seeds(const RepParams& rp, uint32_t step) {
  DevSeedStream& s = rp.sim->rnd;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t x = lane < 31u ? s.st.r[lane] : 0u;
  const uint32_t draw = __shfl_sync(0xffffffffu, x, (lane + 15u) & 31u), before = __shfl_sync(0xffffffffu, x, (lane + 12u) & 31u);
  const uint32_t kept = __shfl_sync(0xffffffffu, x, (lane + 16u) & 31u);  // lanes 16 on: word lane - 16
  if (lane < 31u) s.st.r[lane] = lane < 16u ? draw - before : kept;
  if (lane == 0u) s.next = step;
}

template <class T>
__device__ void load_model_const(const T* g, T& s) {
  const float* src = reinterpret_cast<const float*>(g);
  float* dst = reinterpret_cast<float*>(&s);
  for (int k = threadIdx.x; k < (int)(sizeof(T) / 4); k += blockDim.x) dst[k] = src[k];
}

// Exclusive scan of one value per thread over the CTA (blockDim.x a multiple
// of 32); s_w holds 33 words. Ends with all threads synchronised.
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_w, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_w[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < nw ? s_w[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    s_w[lane] = wi - w;
    if (lane == 31) s_w[32] = wi;
  }
  __syncthreads();
  const uint32_t r = s_w[warp] + incl - v;
  *total = s_w[32];
  __syncthreads();
  return r;
}

// Ticket ranges of a pass over the batch: replicate r owns tickets
// [s_pre[r], s_pre[r+1]); s_pre[nrep] is the number of tickets. tiles(r) is
// r's tile count in this pass. All threads; ends synchronised.
template <class F>
__device__ void plan_tickets(uint32_t nrep, uint32_t* s_pre, uint32_t* s_w, F tiles) {
  if (nrep == 1) {  // a single simulation
    if (threadIdx.x == 0) {
      s_pre[0] = 0;
      s_pre[1] = tiles(0u);
    }
    __syncthreads();
    return;
  }
  const uint32_t per = (nrep + blockDim.x - 1) / blockDim.x;  // <= 4: nrep <= kMaxRep, blockDim.x >= 256
  const uint32_t r0 = min(threadIdx.x * per, nrep), r1 = min(r0 + per, nrep);
  uint32_t loc[4], sum = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    loc[k] = r0 + k < r1 ? tiles(r0 + k) : 0u;
    sum += loc[k];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(sum, s_w, &total);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (r0 + k < r1) s_pre[r0 + k] = run;
    run += loc[k];
  }
  if (threadIdx.x == 0) s_pre[nrep] = total;
  __syncthreads();
}

// The replicate owning ticket t < s_pre[nrep].
__device__ __forceinline__ uint32_t find_rep(const uint32_t* s_pre, uint32_t nrep, uint32_t t) {
  uint32_t lo = 0, hi = nrep;  // s_pre[lo] <= t < s_pre[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (s_pre[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes, int i, int n) {
  const uint4* s = reinterpret_cast<const uint4*>(src);
  uint4* d = reinterpret_cast<uint4*>(dst);
  for (int k = i; k < bytes / 16; k += n) d[k] = s[k];
}
static_assert(sizeof(StepCtx) % 16 == 0, "StepCtx is copied in 16-byte words");

// ------------------------------------------------------------------------
// The two passes of a step
// ------------------------------------------------------------------------
// Both passes cut every active replicate's pool into spans of
// span_size(end) slots and give the spans of the batch to the warps of a
// grid of resident CTAs in turn (warp w takes units w, w + W, ...). A warp
// walks its span range by range, 32 slots of one state at a time, with code
// specialised for the state, and shares nothing with the other warps but the
// span counts, so neither pass has a barrier, a ticket or a staged tile in
// its loop.
//
// What bounds them is the number of instructions per agent and the bytes of
// its record, so both are kept to what the state needs (state_cols): an egg
// or a larva carries its age and delay (hoursInState follows from the age),
// the sporogonic and gonotrophic fields are zero until a female seeks blood,
// and the columns of a field that a state implies are neither read
// nor written. A pool whose loaded records do not obey that (k_pool_stats
// checks) and the caller-owned pools of sampo_step_noalloc take the WIDE
// passes, which move whole records.
constexpr uint32_t kNoRep = 0xffffffffu;

enum : uint32_t {
  C_AGE = 1, C_HIS = 2, C_DELAY = 4, C_SPORO = 8, C_UNI = 16, C_AVAIL = 32, C_CYCLE = 64, C_HBC = 128, C_BATCHES = 256,
  C_ALL = 511
};
// Columns that hold an agent's record in state rg; the others are implied:
// zero, or hoursInState = ageInHours (eggs) and ageInHours - 24 (larvae).
__host__ __device__ constexpr uint32_t state_cols(int rg, bool wide) {
  return wide || rg >= BMS ? (uint32_t)C_ALL
         : rg == EGG       ? (uint32_t)(C_AGE | C_DELAY)
         : rg == LARVA     ? (uint32_t)(C_AGE | C_DELAY | C_UNI)
                           : (uint32_t)(C_AGE | C_HIS | C_DELAY | C_UNI);
}
// Columns the decision part of the update reads (update_agent<false>).
__host__ __device__ constexpr uint32_t decide_cols(int rg, bool wide) {
#ifdef SAMPO_USER_SPECIES
  if (rg == GRAVID) return C_ALL;  // the header's layEggs may read any of the agent's fields
#endif
  return rg == EGG     ? (uint32_t)(C_DELAY | (wide ? C_HIS : C_AGE))
         : rg == LARVA ? (uint32_t)(C_AGE | C_DELAY | C_UNI | (wide ? C_HIS : 0))
         : rg == PUPA  ? (uint32_t)(C_HIS | C_DELAY)
         : rg == GRAVID ? (uint32_t)(C_AGE | C_AVAIL | C_UNI)
                        : (uint32_t)(C_AGE | C_HIS | C_DELAY);
}
__host__ __device__ constexpr uint32_t num_cols(uint32_t cols) {
  uint32_t n = 0;
  for (; cols; cols &= cols - 1u) n++;
  return n;
}

// The columns of a range stream through a ring of chunks in the warp's own
// piece of shared memory (cp.async, 16 bytes per lane), so that the loads of
// the next chunks are in flight while one is worked on and cost no registers
// (without the ring a warp waited a full memory latency for every four rows:
// 57 % of its cycles). The chunk is the largest of 32 * I, 64 or 32 slots of
// which at least two fit (I = 4 or 2, the "slots per thread").
constexpr int kRowUnroll = 2;  // rows of a chunk unrolled together
constexpr uint32_t kRingBytes = 5120;
template <uint32_t COLS, uint32_t BYTE_COLS, int I>
struct Ring {
  static constexpr uint32_t kSlotBytes = 4 * num_cols(COLS) + BYTE_COLS;
  __host__ __device__ static constexpr uint32_t fits(uint32_t slots) { return kRingBytes / (slots * kSlotBytes); }
  static constexpr uint32_t kSlots = (I == 4 && fits(128) >= 2) ? 128u : fits(64) >= 2 ? 64u : 32u;
  static constexpr uint32_t kStages = fits(kSlots) > 4 ? 4u : fits(kSlots);
  static constexpr uint32_t kStageBytes = kSlots * kSlotBytes;
  static_assert(kStages >= 2 && kStageBytes % 16 == 0, "two chunks at least, on 16-byte boundaries");
  __host__ __device__ static constexpr uint32_t offset(uint32_t col) { return num_cols(COLS & (col - 1u)) * kSlots * 4u; }
  static constexpr uint32_t kByteOffset = num_cols(COLS) * kSlots * 4u;
};
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Starts the copies of the chunk at slot g0 (a multiple of 32) into the
// stage: four slots per lane, as far as the range reaches (rounded up to four
// slots, inside the columns' slack).
template <class RING, uint32_t COLS>
__device__ __forceinline__ void issue_chunk(uint8_t* st, const DevPool& s, const uint8_t* bytes0, const uint8_t* bytes1, uint32_t g0, uint32_t hi) {
  const uint32_t i = 4u * (threadIdx.x & 31u);
  const size_t g = (size_t)g0 + i;
  if (i < RING::kSlots && g < hi) {
    if (COLS & C_AGE) cp_async16(st + RING::offset(C_AGE) + 4 * i, s.age + g);
    if (COLS & C_HIS) cp_async16(st + RING::offset(C_HIS) + 4 * i, s.his + g);
    if (COLS & C_DELAY) cp_async16(st + RING::offset(C_DELAY) + 4 * i, s.delay + g);
    if (COLS & C_SPORO) cp_async16(st + RING::offset(C_SPORO) + 4 * i, s.sporo + g);
    if (COLS & C_UNI) cp_async16(st + RING::offset(C_UNI) + 4 * i, s.uni + g);
    if (COLS & C_AVAIL) cp_async16(st + RING::offset(C_AVAIL) + 4 * i, s.avail + g);
    if (COLS & C_CYCLE) cp_async16(st + RING::offset(C_CYCLE) + 4 * i, s.cycle + g);
    if (COLS & C_HBC) cp_async16(st + RING::offset(C_HBC) + 4 * i, s.hbc + g);
    if (COLS & C_BATCHES) cp_async16(st + RING::offset(C_BATCHES) + 4 * i, s.batches + g);
    if (bytes0) cp_async4(st + RING::kByteOffset + i, bytes0 + g);
    if (bytes1) cp_async4(st + RING::kByteOffset + RING::kSlots + i, bytes1 + g);
  }
  cp_async_commit();
}
template <class RING, uint32_t COLS>
__device__ __forceinline__ void read_chunk(const uint8_t* st, uint32_t i, Rec& a) {
  const float* f = reinterpret_cast<const float*>(st) + i;
  const uint32_t* u = reinterpret_cast<const uint32_t*>(st) + i;
  a.age = (COLS & C_AGE) ? f[RING::offset(C_AGE) / 4] : 0.0f;
  a.his = (COLS & C_HIS) ? f[RING::offset(C_HIS) / 4] : 0.0f;
  a.delay = (COLS & C_DELAY) ? f[RING::offset(C_DELAY) / 4] : 0.0f;
  a.sporo = (COLS & C_SPORO) ? f[RING::offset(C_SPORO) / 4] : 0.0f;
  a.uni = (COLS & C_UNI) ? u[RING::offset(C_UNI) / 4] : 0u;
  a.avail = (COLS & C_AVAIL) ? u[RING::offset(C_AVAIL) / 4] : 0u;
  a.cycle = (COLS & C_CYCLE) ? u[RING::offset(C_CYCLE) / 4] : 0u;
  a.hbc = (COLS & C_HBC) ? u[RING::offset(C_HBC) / 4] : 0u;
  a.batches = (COLS & C_BATCHES) ? u[RING::offset(C_BATCHES) / 4] : 0u;
  a.female = 0u;
  a.bm = BM_NONE;
}
// Walks slots [lo, hi) of the current buffer in chunks: f(stage, first slot)
// for each, with the copies of the following chunks in flight. Every lane
// calls it; the stage may be read by any lane until f returns.
template <class RING, uint32_t COLS, class F>
__device__ __forceinline__ void stream_range(uint8_t* ring, const DevPool& s, const uint8_t* bytes0, const uint8_t* bytes1, uint32_t lo,
                                             uint32_t hi, F&& f) {
  constexpr uint32_t N = RING::kStages;
  const uint32_t first = lo & ~31u;
#pragma unroll
  for (uint32_t j = 0; j < N - 1; j++) issue_chunk<RING, COLS>(ring + j * RING::kStageBytes, s, bytes0, bytes1, first + j * RING::kSlots, hi);
  uint32_t rd = 0, wr = N - 1;
  for (uint32_t g0 = first; g0 < hi; g0 += RING::kSlots) {
    issue_chunk<RING, COLS>(ring + wr * RING::kStageBytes, s, bytes0, bytes1, g0 + (N - 1) * RING::kSlots, hi);
    cp_async_wait<N - 1>();
    __syncwarp();  // every lane's copies of this chunk are in
    f(ring + rd * RING::kStageBytes, g0);
    __syncwarp();  // the stage is read before its next copies start
    rd = rd + 1 == N ? 0 : rd + 1;
    wr = wr + 1 == N ? 0 : wr + 1;
  }
  cp_async_wait<0>();
}
// The same columns of one slot, from the pool itself.
template <uint32_t COLS>
__device__ __forceinline__ void load_cols(const DevPool& s, uint32_t g, Rec& a) {
  a.age = (COLS & C_AGE) ? __ldg(s.age + g) : 0.0f;
  a.his = (COLS & C_HIS) ? __ldg(s.his + g) : 0.0f;
  a.delay = (COLS & C_DELAY) ? __ldg(s.delay + g) : 0.0f;
  a.sporo = (COLS & C_SPORO) ? __ldg(s.sporo + g) : 0.0f;
  a.uni = (COLS & C_UNI) ? __ldg(s.uni + g) : 0u;
  a.avail = (COLS & C_AVAIL) ? __ldg(s.avail + g) : 0u;
  a.cycle = (COLS & C_CYCLE) ? __ldg(s.cycle + g) : 0u;
  a.hbc = (COLS & C_HBC) ? __ldg(s.hbc + g) : 0u;
  a.batches = (COLS & C_BATCHES) ? __ldg(s.batches + g) : 0u;
  a.female = 0u;
  a.bm = BM_NONE;
}
// The fields a narrow record implies.
template <int RG, bool WIDE>
__device__ __forceinline__ void implied_fields(Rec& a) {
  if (!WIDE && RG == EGG) a.his = a.age;
  if (!WIDE && RG == LARVA) a.his = a.age - 24.0f;
}
// Stores to a pool that the kernel does not read: as global stores that the
// compiler need not order against the warps' state in shared memory (through
// the pools' pointers, which it reads from memory, it would take them for
// stores to anywhere, and read the step's constants again after each).
__device__ __forceinline__ void put(float* p, float v) { asm volatile("st.global.f32 [%0], %1;" ::"l"(p), "f"(v)); }
__device__ __forceinline__ void put(uint32_t* p, uint32_t v) { asm volatile("st.global.u32 [%0], %1;" ::"l"(p), "r"(v)); }
__device__ __forceinline__ void put(uint8_t* p, uint32_t v) { asm volatile("st.global.u8 [%0], %1;" ::"l"(p), "r"(v)); }
template <uint32_t COLS>
__device__ __forceinline__ void store_cols(const DevPool& d, uint32_t g, const Rec& a) {
  if (COLS & C_AGE) put(d.age + g, a.age);
  if (COLS & C_HIS) put(d.his + g, a.his);
  if (COLS & C_DELAY) put(d.delay + g, a.delay);
  if (COLS & C_SPORO) put(d.sporo + g, a.sporo);
  if (COLS & C_UNI) put(d.uni + g, a.uni);
  if (COLS & C_AVAIL) put(d.avail + g, a.avail);
  if (COLS & C_CYCLE) put(d.cycle + g, a.cycle);
  if (COLS & C_HBC) put(d.hbc + g, a.hbc);
  if (COLS & C_BATCHES) put(d.batches + g, a.batches);
}

// Survivors by next state, 16 bits each: states 0-1, 2-3, 4-5, 6-7. A span
// has at most 2^10 slots and a super (32 spans) 2^15, so no field carries.
__device__ __forceinline__ uint32_t state_count(const uint4& v, int b) {
  const uint32_t w = b < 2 ? v.x : b < 4 ? v.y : b < 6 ? v.z : v.w;
  return (w >> (16 * (b & 1))) & 0xffffu;
}
template <int B>
__device__ __forceinline__ void add_count(uint4& v, uint32_t n) {
  const uint32_t x = n << (16 * (B & 1));
  if (B < 2) v.x += x;
  else if (B < 4) v.y += x;
  else if (B < 6) v.z += x;
  else v.w += x;
}
// One lane: adds a span's counts to its super's.
__device__ __forceinline__ void add_super(uint4* sup, const uint4& v) {
  unsigned long long* q = reinterpret_cast<unsigned long long*>(sup);
  const unsigned long long a = v.x | ((unsigned long long)v.y << 32), b = v.z | ((unsigned long long)v.w << 32);
  if (a) atomicAdd(q, a);
  if (b) atomicAdd(q + 1, b);
}

// Once every span of the replicate is counted: the exclusive prefix by state
// of each super and the totals (cnt, 8 words); the raw counts are cleared for
// the next step. The calling threads (nt of them, thread t) take contiguous
// runs of supers: one pass of independent loads, one scan over the threads
// (`scan` returns a thread's exclusive prefix of a value and the total), one
// pass back.
template <class Scan>
__device__ __forceinline__ void scan_supers(const RepParams& rp, uint32_t nspans, uint32_t* cnt, uint32_t t, uint32_t nt, Scan scan) {
  const uint32_t nsup = (nspans + 31u) / 32u, per = (nsup + nt - 1u) / nt;
  const uint32_t i0 = min(t * per, nsup), i1 = min(i0 + per, nsup);
  uint32_t sum[8];
#pragma unroll
  for (int b = 0; b < 8; b++) sum[b] = 0;
#pragma unroll 4
  for (uint32_t i = i0; i < i1; i++) {
    const uint4 v = __ldcg(rp.supers + i);
#pragma unroll
    for (int b = 0; b < 8; b++) sum[b] += state_count(v, b);
  }
  uint32_t run[8];
  scan(sum, run, cnt);
#pragma unroll 2
  for (uint32_t i = i0; i < i1; i++) {
    const uint4 v = __ldcg(rp.supers + i);
    uint4* o = reinterpret_cast<uint4*>(rp.superPre + (size_t)i * 8);
    o[0] = make_uint4(run[0], run[1], run[2], run[3]);
    o[1] = make_uint4(run[4], run[5], run[6], run[7]);
    rp.supers[i] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int b = 0; b < 8; b++) run[b] += state_count(v, b);
  }
}
// The eight sums of the lanes of a warp: exclusive prefixes; lane 31 has the totals in incl.
__device__ __forceinline__ void warp_scan8(const uint32_t (&sum)[8], uint32_t (&run)[8], uint32_t (&incl)[8]) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    uint32_t x = sum[b];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    incl[b] = x;
    run[b] = x - sum[b];
  }
}
// scan_supers by one warp.
__device__ void scan_supers_warp(const RepParams& rp, uint32_t nspans, uint32_t* cnt) {
  const uint32_t lane = threadIdx.x & 31u;
  scan_supers(rp, nspans, cnt, lane, 32u, [&](const uint32_t (&sum)[8], uint32_t (&run)[8], uint32_t* tot) {
    uint32_t incl[8];
    warp_scan8(sum, run, incl);
    if (lane == 31u) {
#pragma unroll
      for (int b = 0; b < 8; b++) tot[b] = incl[b];
    }
  });
}
// scan_supers by a CTA of at most 32 warps (all threads; ends synchronised).
// s_part: 32 x 8 words.
__device__ void scan_supers_block(const RepParams& rp, uint32_t nspans, uint32_t* cnt, uint32_t (*s_part)[8]) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  scan_supers(rp, nspans, cnt, threadIdx.x, blockDim.x, [&](const uint32_t (&sum)[8], uint32_t (&run)[8], uint32_t* tot) {
    uint32_t incl[8];
    warp_scan8(sum, run, incl);
    if (lane == 31u) {
#pragma unroll
      for (int b = 0; b < 8; b++) s_part[warp][b] = incl[b];
    }
    __syncthreads();
    if (threadIdx.x < 8) {  // one state per thread over the warps
      uint32_t x = 0;
      for (uint32_t i = 0; i < nw; i++) {
        const uint32_t y = s_part[i][threadIdx.x];
        s_part[i][threadIdx.x] = x;
        x += y;
      }
      tot[threadIdx.x] = x;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 8; b++) run[b] += s_part[warp][b];
  });
  __syncthreads();
}

// The kernels of a batch's hour are launched with programmatic serialisation:
// the CTAs of a pass come up while k_publish still runs, and wait here for its
// end (and with it that of all before) before they read anything it wrote.
// (The passes do not let k_publish come up early: 2 % slower, its CTAs then
// wait for room between theirs.)
__device__ __forceinline__ void wait_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void start_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What a warp holds of the replicate its unit belongs to; reloaded only when
// its next unit belongs to another one.
struct alignas(16) WarpRep {
  StepCtx c;                    // constants of the step
  StepCtx c1;                   // and of the step after, in a pass that decides ahead
  uint32_t larvaKill1[100];     // its larval mortality
  sampo_population pop, next;   // current ranges; the next pool's (update/scatter pass)
  DevPool src, dst;
  uint8_t* dec;                 // decisions of caller-owned pools, or null: in the flags
  uint4 *spans, *spans1, *spans2;  // span counts of the step, of the step after, and the ones to clear
  uint4* supers;
  const uint32_t* superPre;
  uint32_t span, nspans, newEggs, ahead;  // slots per span, spans, eggs laid, whether it decides ahead
  uint32_t span1, clear, clearPer;        // slots per span of the next pool; spans to clear, and of them per unit
};
// Words of src to dst by the lanes of a warp.
template <class T>
__device__ __forceinline__ void warp_copy(T* dst, const T* src) {
  static_assert(sizeof(T) % 4 == 0, "whole words");
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  const uint32_t* q = reinterpret_cast<const uint32_t*>(src);
  for (int k = threadIdx.x & 31; k < (int)(sizeof(T) / 4); k += 32) d[k] = q[k];
}
// (PASS2: also what the update/scatter pass needs)
template <bool PASS2, bool AHEAD>
__device__ __forceinline__ void load_warp_rep(const RepParams& rp, uint32_t min_span, WarpRep& w) {
  const SimDev* sim = rp.sim;
  const uint32_t cur = sim->cur, par = sim->step & 1u;
  __syncwarp();  // every lane is past its reads of the last replicate's
  warp_copy(&w.c, &sim->ctx[par]);
  if (AHEAD) {
    // a replicate that stops after this step decides nothing ahead: it runs
    // through the same code with this step's constants, and nothing is kept
    const uint32_t q = sim->ahead ? par ^ 1u : par;
    warp_copy(&w.c1, &sim->ctx[q]);
    for (uint32_t k = threadIdx.x & 31; k < 100; k += 32) w.larvaKill1[k] = sim->larvaKill[q][k];
  }
  warp_copy(&w.pop, &sim->pop);
  warp_copy(&w.src, &rp.pool[cur]);
  if (PASS2) warp_copy(&w.dst, &rp.pool[cur ^ 1u]);
  if ((threadIdx.x & 31) == 0) {
    const uint32_t end = sim->pop.r[GRAVID].end, rot = sim->rot;
    w.dec = rp.dec;
    w.spans = rp.spans + (size_t)rot * rp.spanStride;
    w.supers = rp.supers;
    w.superPre = rp.superPre;
    w.span = span_size(end, min_span);
    w.nspans = units_of(end, w.span);
    w.newEggs = sim->dec.newEggs;
    if (PASS2) {
      uint32_t tc[8], base[8];
      for (int k = 0; k < 8; k++) tc[k] = sim->cnt[k];
      sampo_population np;
      next_layout(tc, w.newEggs, np, base);
      w.next = np;
      if (AHEAD) {
        w.ahead = sim->ahead;
        w.span1 = span_size(np.r[GRAVID].end, min_span);
        w.spans1 = rp.spans + (size_t)(rot == 2u ? 0u : rot + 1u) * rp.spanStride;
        const uint32_t old = rot == 0u ? 2u : rot - 1u, units = w.nspans + units_of(w.newEggs, w.span);
        w.spans2 = rp.spans + (size_t)old * rp.spanStride;
        w.clear = w.ahead ? min(sim->dirty[old], rp.spanStride) : 0u;  // (no store leaves the set)
        w.clearPer = units ? (w.clear + units - 1u) / units : 0u;
      }
    }
  }
  __syncwarp();
}

// Slots whose agents move on to another state this hour wait here until 32
// are there (or the range ends) and are then written out by 32 lanes at once:
// in a row of 32 agents one moves every few hours, and its transition (for a
// hatching egg a normal draw) would occupy the warp for a single lane. A
// power of two above 31 + a chunk's slots.
constexpr uint32_t kMoved = 256;

// What a warp adds to its replicate, gathered range by range in shared memory
// (written by lane 0).
struct WarpSum {
  Decided dec;                 // of the step being decided
  uint32_t fem, inf, bnc[4];   // of the pool being written
  uint32_t error;
  uint32_t rep, spans;         // the replicate they belong to; count pass: spans counted
};
__device__ __forceinline__ void clear_sum(WarpSum& t) {
  t.dec = Decided{0u, 0u, 0xffffffffu, 0u};
  t.fem = t.inf = t.error = 0;
  t.bnc[0] = t.bnc[1] = t.bnc[2] = t.bnc[3] = 0;
}
// Lane 0: the warp's sums into its replicate, and cleared.
__device__ __forceinline__ void flush_sum(WarpSum& t, SimDev* sim, Decided* to) {
  if (t.dec.newEggs) atomicAdd(&to->newEggs, t.dec.newEggs);
  if (t.dec.L1de) atomicAdd(&to->L1de, t.dec.L1de);
  if (t.dec.dmin != 0xffffffffu) { atomicMin(&to->dmin, t.dec.dmin); atomicMax(&to->dmax, t.dec.dmax); }
  if (t.fem) atomicAdd(&sim->acc_fem, t.fem);
  if (t.inf) atomicAdd(&sim->acc_inf, t.inf);
  for (int j = 0; j < 4; j++)
    if (t.bnc[j]) atomicAdd(&sim->acc_bnc[j], t.bnc[j]);
  if (t.error) atomicOr(&sim->error, t.error);
  clear_sum(t);
}

// The end of a pass (every thread of the CTA): the sums that its warps hold
// (WarpSum::rep) into their replicates', the CTA's warps of one replicate
// together (the adds of 3,648 warps to the same few words, all at the end,
// queued up: k_scatter 113 -> 109 us at 5e6 caller-owned agents). Returns, on the lanes of the first warp of a
// replicate, the spans its warps have counted (0 on other warps).
__device__ __forceinline__ uint32_t flush_sums(const RepParams* reps, WarpSum* sums, bool dec_ahead) {
  constexpr uint32_t kMin = 2, kMax = 3, kFem = 4, kBnc = 6, kError = 10, kSpans = 12;  // a WarpSum's words
#ifndef __CUDACC_RTC__  // (it has no offsetof)
  static_assert(offsetof(WarpSum, dec.dmin) == 4 * kMin && offsetof(WarpSum, dec.dmax) == 4 * kMax && offsetof(WarpSum, fem) == 4 * kFem &&
                offsetof(WarpSum, bnc) == 4 * kBnc && offsetof(WarpSum, error) == 4 * kError && offsetof(WarpSum, spans) == 4 * kSpans &&
                offsetof(SimDev, acc_inf) == offsetof(SimDev, acc_fem) + 4, "words of the sums");
#endif
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  __syncthreads();
  const uint32_t rep = sums[warp].rep;
  for (uint32_t j = 0; j < warp; j++)
    if (sums[j].rep == rep) return 0u;
  if (rep == kNoRep) return 0u;
  const uint32_t k = min(lane, kSpans);
  uint32_t sum = 0, lo = 0xffffffffu, hi = 0, any = 0;
#pragma unroll
  for (uint32_t j = 0; j < kWarps; j++) {
    if (sums[j].rep != rep) continue;
    const uint32_t x = reinterpret_cast<const uint32_t*>(&sums[j])[k];
    sum += x;
    lo = min(lo, x);
    hi = max(hi, x);
    any |= x;
  }
  SimDev* sim = reps[rep].sim;
  uint32_t* dec = reinterpret_cast<uint32_t*>(dec_ahead ? &sim->ahead_dec : &sim->dec);
  if (lane == kMin) {
    if (lo != 0xffffffffu) atomicMin(dec + kMin, lo);
  } else if (lane == kMax) {
    if (hi) atomicMax(dec + kMax, hi);
  } else if (lane < kFem) {
    if (sum) atomicAdd(dec + lane, sum);
  } else if (lane < kBnc) {
    if (sum) atomicAdd(&sim->acc_fem + (lane - kFem), sum);
  } else if (lane < kError) {
    if (sum) atomicAdd(&sim->acc_bnc[lane - kBnc], sum);
  } else if (lane == kError) {
    if (any) atomicOr(&sim->error, any);
  }
  return __shfl_sync(0xffffffffu, sum, kSpans);
}

// The dynamic shared memory of the two passes, followed by the batch's unit
// prefix (nrep + 1 words, sized at launch so that a single simulation pays 8
// bytes for it). The code of a range is a function of its own, so that its
// registers are its own (inlined together, the eight ranges' code spilled in
// its loops); it finds its warp's state here.
struct alignas(128) PassShared {
  uint8_t ring[kWarps][kRingBytes];
  WarpRep rep[kWarps];
  ModelConst mc;
  uint32_t moved[kWarps][kMoved];
  WarpSum sum[kWarps];
  uint32_t scan[36];
};
extern __shared__ __align__(128) uint8_t pass_shared_memory[];
__device__ __forceinline__ PassShared& pass_shared() { return *reinterpret_cast<PassShared*>(pass_shared_memory); }
__host__ __device__ constexpr size_t pass_smem(uint32_t nrep) {
  return sizeof(PassShared) + (((size_t)(nrep + 1) * 4 + 15) & ~(size_t)15);
}

// What a lane's decisions in one range add up to.
struct DecideAcc {
  Acc acc;             // newEggs and bad
  uint32_t l1, dmin, dmax, devoob;
};
__device__ __forceinline__ void clear_acc(DecideAcc& d) {
  d.acc = Acc{0, 0, 0, 0, 0, 0};
  d.l1 = d.dmax = d.devoob = 0;
  d.dmin = 0xffffffffu;
}
// A range's decisions (state RG, and NX for those that moved there) into the warp's sums.
template <int RG, int NX>
__device__ __forceinline__ void add_decided(const DecideAcc& d, WarpSum& t) {
  constexpr bool larvae = RG <= LARVA || NX == LARVA, lays = RG == GRAVID || NX == GRAVID;
  const uint32_t ne = lays ? __reduce_add_sync(0xffffffffu, d.acc.newEggs) : 0u;
  const uint32_t l1 = larvae ? __reduce_add_sync(0xffffffffu, d.l1) : 0u;
  const uint32_t mn = larvae ? __reduce_min_sync(0xffffffffu, d.dmin) : 0xffffffffu, mx = larvae ? __reduce_max_sync(0xffffffffu, d.dmax) : 0u;
  const uint32_t bad = larvae ? __reduce_or_sync(0xffffffffu, (d.acc.bad ? SAMPO_DEV_ERR_LARVATABLE : 0u) |
                                                                (d.devoob ? SAMPO_DEV_ERR_DEVRATES : 0u)) : 0u;
  if ((threadIdx.x & 31) == 0) {
    t.dec.newEggs += ne;
    t.dec.L1de += l1;
    t.dec.dmin = min(t.dec.dmin, mn);
    t.dec.dmax = max(t.dec.dmax, mx);
    t.error |= bad;
  }
}
// A range's (or its moves') females and counters into the warp's sums.
template <int RG>
__device__ __forceinline__ void add_moved(uint32_t fem, uint32_t inf, const Acc& acc, WarpSum& t) {
  uint32_t v[6] = {fem, inf, acc.cycles, acc.sumCycles, acc.bites, acc.infectBites};
#pragma unroll
  for (int j = 0; j < 6; j++) v[j] = (j < 2 || RG >= BMS) ? __reduce_add_sync(0xffffffffu, v[j]) : 0u;
  if ((threadIdx.x & 31) == 0) {
    t.fem += v[0];
    t.inf += v[1];
#pragma unroll
    for (int j = 0; j < 4; j++) t.bnc[j] += v[2 + j];
  }
}
// The decision about the agent a at slot g of range RG (a: its fields of
// decide_cols; changed). Adds the larva it leaves to the next pool's
// statistics (kernel/calcL1de.cl:28-30).
template <int RG, bool WIDE>
__device__ __forceinline__ uint32_t decide(const StepCtx& c, const KillConst& kc, uint32_t g, Rec& a, DecideAcc& d) {
  if (RG == LARVA) d.devoob |= c.devOOB;
  const uint32_t code = decision_code(RG, update_agent<false, true, true, false, !WIDE>(c, kc, RG, g, a, d.acc));
  if (RG == EGG && code == DEC_MOVES) {  // hatched: 24 hours old
    d.l1 += 1u;
    d.dmin = min(d.dmin, 1u); d.dmax = max(d.dmax, 1u);
  }
  if (RG == LARVA && code == DEC_STAYS) {
    const uint32_t dd = age_days<!WIDE>(a.age);
    d.l1 += age_days_uncapped<!WIDE>(a.age);
    d.dmin = min(d.dmin, dd); d.dmax = max(d.dmax, dd);
  }
  return code;
}

// The count pass over slots [lo, hi) of range RG: each agent's decision into
// its flags (bits 4-5), or into dec where the pool belongs to the caller.
// Returns the agents that stay | those that move on << 16 (a span has at most
// 2^10).
template <int I, bool WIDE, int RG>
__device__ __noinline__ uint32_t count_range(uint32_t lo, uint32_t hi) {
  PassShared& ps = pass_shared();
  const uint32_t warp = threadIdx.x >> 5;
  const WarpRep& w = ps.rep[warp];
  const KillConst& kc = ps.mc.kill;
  constexpr uint32_t COLS = decide_cols(RG, WIDE);
  using RING = Ring<COLS, 1, I>;
  const uint32_t lane = threadIdx.x & 31u;
  const DevPool src = w.src;
  uint8_t* const dec = WIDE ? w.dec : nullptr;
  const StepCtx& c = w.c;
  DecideAcc da;
  clear_acc(da);
  uint32_t ns_stay = 0, ns_move = 0;
  stream_range<RING, COLS>(ps.ring[warp], src, src.flags, nullptr, lo, hi, [&](const uint8_t* st, uint32_t g0) {
#pragma unroll kRowUnroll
    for (uint32_t k = 0; k < RING::kSlots / 32; k++) {
      const uint32_t i = 32u * k + lane, g = g0 + i;
      uint32_t code = DEC_DIES;
      if (g >= lo && g < hi) {
        Rec a;
        read_chunk<RING, COLS>(st, i, a);
        const uint32_t fl = st[RING::kByteOffset + i];
        implied_fields<RG, WIDE>(a);
        a.female = (fl >> 3) & 1u;
        code = decide<RG, WIDE>(c, kc, g, a, da);
        if (WIDE && dec) put(dec + g, code);
        else put(src.flags + g, (fl & 15u) | (code << 4));
      }
      ns_stay += __popc(__ballot_sync(0xffffffffu, code == DEC_STAYS));
      ns_move += __popc(__ballot_sync(0xffffffffu, code == DEC_MOVES));
    }
  });
  add_decided<RG, RG>(da, ps.sum[warp]);
  return ns_stay | (ns_move << 16);
}

// Calls f<RG>(lo, hi) for the part of every range that lies in [u0, u1), in
// slot order.
template <int RG = 0, class F>
__device__ __forceinline__ void for_ranges(const sampo_population& pop, uint32_t u0, uint32_t u1, F&& f) {
  if constexpr (RG < NSTATE) {
    const uint32_t lo = max(pop.r[RG].start, u0), hi = min(pop.r[RG].end, u1);
    if (lo < hi) f.template operator()<RG>(lo, hi);
    for_ranges<RG + 1>(pop, u0, u1, f);
  }
}

template <int I, bool WIDE>
struct CountRanges {
  uint4& cs;
  template <int RG>
  __device__ __forceinline__ void operator()(uint32_t lo, uint32_t hi) {
    const uint32_t n = count_range<I, WIDE, RG>(lo, hi);
    add_count<RG>(cs, n & 0xffffu);
    add_count<next_state(RG)>(cs, n >> 16);
  }
};

// The count pass: decisions, the survivors by next state of every span and
// super, and (by the warp that finishes the replicate's last span) the
// supers' prefixes and the replicate's totals. Spans are taken from the last
// one down, so that the update/scatter pass starts on those this pass
// touched last.
template <int I, bool WIDE>
__global__ void __launch_bounds__(kBlock, 3) k_count(KParams p) {
  PassShared& ps = pass_shared();
  uint32_t* s_pre = reinterpret_cast<uint32_t*>(pass_shared_memory + sizeof(PassShared));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  load_model_const(&p.mc->kill, ps.mc.kill);
  wait_previous_kernel();
  const uint32_t min_span = p.bat->minSpan;
  plan_tickets(p.nrep, s_pre, ps.scan, [&](uint32_t r) -> uint32_t {
    const SimDev* sim = p.reps[r].sim;
    return sim->active ? span_count(sim->pop.r[GRAVID].end, min_span) : 0u;
  });
  __syncthreads();
  const uint32_t total = s_pre[p.nrep], stride = gridDim.x * kWarps;
  WarpRep& w = ps.rep[warp];
  WarpSum& sum = ps.sum[warp];
  if (lane == 0) clear_sum(sum);
  uint32_t cur_rep = kNoRep, done = 0;
  // `n` counted spans into the replicate's: the warp that brings the last ones scans the supers
  auto arrive = [&](uint32_t n) {
    const RepParams& rp = p.reps[cur_rep];
    SimDev* sim = rp.sim;
    uint32_t last = 0;
    if (lane == 0) {
      __threadfence();  // the adds to the supers come before the arrival
      last = atomicAdd(&sim->spans_done, n) + n == w.nspans;
      __threadfence();
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();
    if (last) {
      scan_supers_warp(rp, w.nspans, sim->cnt);
      if (lane == 0) {
        sim->spans_done = 0;
        sim->dirty[sim->rot] = max(sim->dirty[sim->rot], w.nspans);
      }
    }
  };
  for (uint32_t u = blockIdx.x * kWarps + warp; u < total; u += stride) {
    const uint32_t t = total - 1u - u;
    const uint32_t r = find_rep(s_pre, p.nrep, t);
    if (r != cur_rep) {  // uniform
      if (cur_rep != kNoRep) {
        if (lane == 0) flush_sum(sum, p.reps[cur_rep].sim, &p.reps[cur_rep].sim->dec);
        arrive(done);
        done = 0;
      }
      load_warp_rep<false, false>(p.reps[r], min_span, w);
      cur_rep = r;
    }
    const uint32_t sp = t - s_pre[r], end = w.pop.r[GRAVID].end, u0 = sp * w.span;
    const uint32_t u1 = end - u0 > w.span ? u0 + w.span : end;
    uint4 cs = make_uint4(0u, 0u, 0u, 0u);
    for_ranges(w.pop, u0, u1, CountRanges<I, WIDE>{cs});
    if (lane == 0) {
      w.spans[sp] = cs;
      add_super(w.supers + (sp >> 5), cs);
    }
    done++;
  }
  if (lane == 0) {
    sum.rep = cur_rep;
    sum.spans = done;
    __threadfence();  // (the first warp of the replicate arrives for this one)
  }
  const uint32_t n = flush_sums(p.reps, ps.sum, false);
  if (n) arrive(n);
}

// ------------------------------------------------------------------------
// Publishing the start of a step
// ------------------------------------------------------------------------
// warp 0 publishes; the other warps fill the 100 entries of the larval table
constexpr int kPublishThreads = 256;
// Supers that warp 0 scans alone (four per lane), while the others fill the
// table; more are scanned by the CTA first.
constexpr uint32_t kScanByWarp = 128;

// The larval hourly mortality of larvae d days old in a pool of L1de l1
// (kernel/killAgents.cl:117-125), as a kill_threshold; 0 outside the ages
// [dmin, dmax] present. In binary32 with the exact result: the binary64
// exp, log and pow of the definition are a serial chain that every CTA's
// entry waited for once an hour (k_step_small 9.7 -> 7.7 us per hour at 1e3
// eggs, 15.3 -> 13.5 over a year from 1e4).
__device__ __forceinline__ uint32_t larva_kill_entry(uint32_t d, uint32_t dmin, uint32_t dmax, uint32_t l1, float cc) {
  if (d < dmin || d > dmax) return 0u;
  return kill_threshold(sampo_larva_hmr((float)l1 / ((float)d * cc * 1.0f)));
}

// A replicate whose decided step does not fit: inactive, the step's counters cleared.
__device__ __forceinline__ void pause_rep(SimDev* sim) {
#pragma unroll
  for (int k = 0; k < 8; k++) sim->cnt[k] = 0;
  sim->dec = Decided{0u, 0u, 0xffffffffu, 0u};
  sim->ahead_dec = Decided{0u, 0u, 0xffffffffu, 0u};
  sim->acc_fem = 0; sim->acc_inf = 0;
  sim->acc_bnc[0] = sim->acc_bnc[1] = sim->acc_bnc[2] = sim->acc_bnc[3] = 0;
  sim->ahead = 0;
  sim->active = 0;
}

// The publish of replicate r by the calling CTA (kPublishThreads threads; all
// of them call it). Step s is the one the replicate is at.
//  PUB_AFTER_STEP  ends step s: the next layout from its survivor counts
//    (kernel/oldToNewAgents.cl:57-95), the pool's L1de, female and infective
//    counts (calcStats, src/abms.c:230-310) and the stats row of s + 1. When
//    the pass decided s + 1 as well, the counts of s + 1 are scanned and
//    become the decided ones.
//  PUB_DECIDED     follows the count pass of step s.
//  PUB_INITIAL     the statistics and row of a pool put in place by the host.
//  PUB_REFRESH     recomputes the input-dependent constants of step s only
//    (its inputs may have been written after its publish).
// Every mode prepares the constants and the larval mortality table
// (kernel/killAgents.cl:117-133 depends on the age and L1de only) of the next
// step somebody decides: the coming step, or with PUB_AHEAD, for a replicate
// that does not stop there, the one after, whose pool's size and L1de the
// decisions already give.
// When the decided step's layout does not fit the replicate's capacity, the
// replicate pauses: it becomes inactive at that step with its pool, constants,
// larval table and seed stream as they are, and only the step's counters are cleared, so
// that the step runs again, with the same result, once its pool has been
// moved into a larger one (sampo_batch_grow).
__device__ void publish_rep(const KParams& p, uint32_t r, int mode_bits) {
  __shared__ uint32_t s_cnt[8], s_part[32][8], s_pause;
  const int mode = mode_bits & PUB_MODE;
  const RepParams& rp = p.reps[r];
  SimDev* sim = rp.sim;
  const uint32_t tid = threadIdx.x;
  if (!sim->active) return;
  const uint32_t s = sim->step, stop = sim->stop_step;
  const bool after = mode == PUB_AFTER_STEP;
  const bool decided = mode == PUB_DECIDED || (after && sim->ahead);  // step sd's decisions are there
  const uint32_t sd = after ? s + 1u : s;                              // the step the replicate is at after this publish
  const bool ahead = decided && (mode_bits & PUB_AHEAD) && sd + 1u < stop;
  const bool prepare = !decided || ahead;      // constants and table of step x
  const uint32_t x = decided ? sd + 1u : sd;
  bool drew = false;  // (warp 0)
  if (tid < 32 && prepare) {
    // a device seed stream draws a step's seeds once, before thread 0 reads
    // them; a replicate that turns out to pause gives them back
    drew = sim->rnd.next == x && x < stop;
    if (drew) draw_step_seeds(rp, x);
    __syncwarp();
  }
  if (mode == PUB_REFRESH) {
    if (tid == 0) {
      CtxInputs in;
      load_ctx_inputs(rp, s, in);
      StepCtx c;
      make_ctx(in, sim->larvaKill[s & 1u], sim->pop, c);
      sim->ctx[s & 1u] = c;
    }
    return;
  }
  const uint32_t min_span = p.bat->minSpan;
  // the decisions whose totals describe the larvae of pool x, and the supers to scan
  const Decided* from = after && decided ? &sim->ahead_dec : &sim->dec;
  const uint32_t l1 = from->L1de, dmin = from->dmin, dmax = from->dmax;
  const float cc = sim->cc;
  // Thread 0 reads all it needs before its first store (a store that may
  // alias a later load would hold that load back until the store is issued,
  // turning the reads into a chain).
  sampo_population np;   // the pool of step sd
  sampo_bites_cycles bnc;
  Decided dec;           // of the step that ends (after), then of step sd
  CtxInputs in;
  uint32_t cnt[8], cur = 0, rot = 0, warn = 0, capacity = 0, nspans = 0, dirty = 0;
  bool shared_end_warn = false, pause = false;
  if (tid == 0) {
    np = sim->pop;
    bnc = sim->bnc;
    dec = sim->dec;
#pragma unroll
    for (int k = 0; k < 8; k++) cnt[k] = sim->cnt[k];
    capacity = sim->capacity;
    cur = sim->cur;
    rot = sim->rot;
    warn = sim->warn;
    const uint32_t fem = sim->acc_fem, inf = sim->acc_inf;
    uint32_t abnc[4];
#pragma unroll
    for (int q = 0; q < 4; q++) abnc[q] = sim->acc_bnc[q];
    if (prepare) load_ctx_inputs(rp, x, in);
    if (after) {
      // the reference's shared empty initial ranges (src/abms.c:204-219) make
      // oldToNewAgents read one prefix-sum entry for several range ends
      bool shared_end = false;
      uint32_t moved = 0;
      for (int k = 1; k < 8; k++) {
        shared_end |= np.r[k].end == np.r[k - 1].end;
        moved += cnt[k];
      }
      shared_end_warn = shared_end && moved;
      pause = !layout_fits(cnt, dec.newEggs, capacity);  // the scatter pass flagged the capacity error and wrote nothing
      if (!pause) {
        nspans = span_count(np.r[GRAVID].end, min_span);  // (of the pool that the step left)
        uint32_t base[8];
        next_layout(cnt, dec.newEggs, np, base);
      }
      bnc.numCyclesReported = abnc[0];
      bnc.sumCyclesReported = abnc[1];
      bnc.numBitesReported = abnc[2];
      bnc.numInfectBitesReported = abnc[3];
    }
    if (mode != PUB_DECIDED) {
      np.numLarvae1DayEquiv = (np.r[LARVA].end > np.r[LARVA].start) ? dec.L1de : 0u;  // kernel/calcL1de.cl:259-280
      np.numFemale = fem;
      np.numPotentiallyInfective = inf;
    }
    if (after && decided) {
      const uint32_t units = nspans + dec.newEggs;  // (the pass cleared the oldest span counts if it had any unit)
      dirty = units ? 0u : sim->dirty[rot == 0u ? 2u : rot - 1u];
      s_part[0][0] = span_count(np.r[GRAVID].end, min_span);
    }
    s_pause = pause;
  }
  __syncthreads();
  if (s_pause) {
    if (tid < 32 && drew) undraw_step_seeds(rp, x);
    if (tid == 0) pause_rep(sim);
    return;
  }
  if (after && decided) {  // the counts of step sd, made while step s was applied
    const uint32_t n = s_part[0][0];
    __syncthreads();
    if ((n + 31u) / 32u > kScanByWarp) scan_supers_block(rp, n, s_cnt, s_part);
    else if (tid < 32) scan_supers_warp(rp, n, s_cnt);
    __syncwarp();
  }
  if (tid == 0) {
    if (after) {
      if (shared_end_warn) sim->warn = warn | SAMPO_DEV_WARN_REF_LAYOUT;
      sim->cur = cur ^ 1u;
      sim->step = sd;
      sim->bnc = bnc;
      if (sd >= stop) sim->active = 0;
    }
    if (mode != PUB_DECIDED) {
      sim->pop = np;
      sampo_stats_row row;
      row.pop = np;
      row.bnc = bnc;
      rp.rows[sd % rp.ring] = row;
      sim->acc_fem = 0; sim->acc_inf = 0;
      sim->acc_bnc[0] = sim->acc_bnc[1] = sim->acc_bnc[2] = sim->acc_bnc[3] = 0;
    }
    sampo_population px = np;  // the pool of step x
    if (after && decided) {
      const uint32_t old = rot == 0u ? 2u : rot - 1u, now = rot == 2u ? 0u : rot + 1u;
      sim->rot = now;
      sim->dirty[old] = dirty;
      sim->dirty[now] = max(sim->dirty[now], span_count(np.r[GRAVID].end, min_span));
      dec = sim->ahead_dec;
      sim->dec = dec;
#pragma unroll
      for (int k = 0; k < 8; k++) sim->cnt[k] = cnt[k] = s_cnt[k];
    } else if (mode != PUB_DECIDED) {
#pragma unroll
      for (int k = 0; k < 8; k++) sim->cnt[k] = 0;
      sim->dec = Decided{0u, 0u, 0xffffffffu, 0u};
    }
    if (after) sim->ahead_dec = Decided{0u, 0u, 0xffffffffu, 0u};
    if (decided) {
      if (!layout_fits(cnt, dec.newEggs, capacity)) {
        atomicOr(&sim->error, SAMPO_DEV_ERR_CAPACITY);
        pause_rep(sim);
        pause = true;
      } else if (ahead) {
        uint32_t base[8];
        next_layout(cnt, dec.newEggs, px, base);
        px.numLarvae1DayEquiv = (px.r[LARVA].end > px.r[LARVA].start) ? dec.L1de : 0u;
      }
    }
    sim->ahead = ahead && !pause ? 1u : 0u;
    if (prepare && !pause) {
      StepCtx c;
      make_ctx(in, sim->larvaKill[x & 1u], px, c);
      sim->ctx[x & 1u] = c;
    }
  } else if (tid >= 32 && prepare) {
    // (a replicate that pauses keeps the table of its step: x is the step after)
    for (uint32_t d = tid - 32; d < 100; d += blockDim.x - 32) sim->larvaKill[x & 1u][d] = larva_kill_entry(d, dmin, dmax, l1, cc);
  }
  if (tid < 32 && drew && __shfl_sync(0xffffffffu, pause, 0)) undraw_step_seeds(rp, x);
}

// The start of one hour called on its own: its inputs, which come with the
// launch (no copies ahead of it in the stream), into their ring slots, and the
// step's constants; the step's row goes beside the status words, so that one
// copy brings both to the host. One thread: what it does is a chain anyway.
__global__ void k_begin_step(KParams p, CtxInputs in, uint32_t slot) {
  if (threadIdx.x != 0) return;
  const RepParams& rp = p.reps[0];
  SimDev* sim = rp.sim;
  rp.T[slot] = in.T;
  rp.env[slot] = in.env;
  rp.wt[slot] = in.wt;
#pragma unroll
  for (int k = 0; k < 4; k++) rp.seeds[(size_t)slot * 4 + k] = in.sd[k];
  sim->begun = rp.rows[slot];
  if (!sim->active) return;
  const uint32_t s = sim->step;
  StepCtx c;
  make_ctx(in, sim->larvaKill[s & 1u], sim->pop, c);
  sim->ctx[s & 1u] = c;
}

// Publishing the start of a step for every replicate of p (one CTA each).
__global__ void __launch_bounds__(kPublishThreads) k_publish(KParams p, int mode) {
  wait_previous_kernel();
  start_next_kernel();
  publish_rep(p, blockIdx.x, mode);
}

// ------------------------------------------------------------------------
// Update + scatter pass
// ------------------------------------------------------------------------
// Deciding ahead: the decisions about survivors that a warp has put into
// consecutive slots of state ST, gathered per span of the next pool: the span
// being counted, the first slot past it, and each lane's counts so far
// (stays | moves on << 16).
struct Tally { uint32_t span, end, cnt; };
__device__ __forceinline__ uint32_t tally_count(uint32_t code) {
  return code == DEC_STAYS ? 1u : code == DEC_MOVES ? 1u << 16 : 0u;
}
template <int ST>
__device__ __forceinline__ void flush_tally(const WarpRep& w, Tally& t) {
  const uint32_t n = __reduce_add_sync(0xffffffffu, t.cnt);
  if (w.ahead && n && (threadIdx.x & 31) == 0) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    add_count<ST>(v, n & 0xffffu);
    add_count<next_state(ST)>(v, n >> 16);
    add_super(w.spans1 + t.span, v);
    add_super(w.supers + (t.span >> 5), v);
  }
  t.cnt = 0;
}
// Starts (slots from `first` on) or continues past t.end.
template <int ST>
__device__ __forceinline__ void next_tally(const WarpRep& w, Tally& t, uint32_t first) {
  if (t.end) flush_tally<ST>(w, t);
  t.span = first / w.span1;
  t.end = (t.span + 1u) * w.span1;
}
// The slots [first, first + n) of a row (n <= 32, so at most two spans); d: a
// lane's slot, c: its tally_count (0 on lanes that hold none).
template <int ST>
__device__ __forceinline__ void add_tally(const WarpRep& w, Tally& t, uint32_t first, uint32_t n, uint32_t d, uint32_t c) {
  if (first >= t.end) next_tally<ST>(w, t, first);
  if (first + n > t.end) {
    const bool here = d < t.end;
    t.cnt += here ? c : 0u;
    next_tally<ST>(w, t, t.end);
    c = here ? 0u : c;
  }
  t.cnt += c;
}

// Lanes where `on` holds store their survivor's narrow egg or larva record.
template <int RG>
__device__ __forceinline__ void put_if(bool on, const DevPool& p, uint32_t d, float age, float delay, float cld, uint32_t flags) {
  if (RG == EGG)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %6, 0;\n\t@p st.global.f32 [%0], %3;\n\t@p st.global.f32 [%1], %4;\n\t@p st.global.u8 [%2], %5;\n\t}"
                 ::"l"(p.age + d), "l"(p.delay + d), "l"(p.flags + d), "f"(age), "f"(delay), "r"(flags), "r"((uint32_t)on));
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %8, 0;\n\t@p st.global.f32 [%0], %4;\n\t@p st.global.f32 [%1], %5;\n\t@p st.global.f32 [%2], %6;\n\t@p st.global.u8 [%3], %7;\n\t}"
                 ::"l"(p.age + d), "l"(p.delay + d), "l"(p.uni + d), "l"(p.flags + d), "f"(age), "f"(delay), "f"(cld), "r"(flags), "r"((uint32_t)on));
}

// The first n of the warp's waiting slots (moved), whose agents of range RG
// move on to the next state: 32 at a time to the slots from bm on. Returns
// the slot after the last. (A function of its own: called once in a span or
// two, it would otherwise take the registers of the rows' loop.)
template <bool WIDE, bool AHEAD, int RG>
__device__ __noinline__ uint32_t move_on(uint32_t n, uint32_t bm) {
  constexpr int NX = next_state(RG);
  constexpr uint32_t CS = state_cols(RG, WIDE), CM = state_cols(NX, WIDE);
  PassShared& ps = pass_shared();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const WarpRep& w = ps.rep[warp];
  const ModelConst& mc = ps.mc;
  WarpSum& sum = ps.sum[warp];
  if (bm + n > w.next.r[NX].end) {  // no store leaves the state's run
    if (lane == 0) sum.error |= SAMPO_DEV_ERR_TILECOUNT;
    return bm;
  }
  Acc acc = {0, 0, 0, 0, 0, 0};
  DecideAcc da;
  clear_acc(da);
  Tally t = {0, 0, 0};
  uint32_t fem = 0, inf = 0;
#pragma unroll 1
  for (uint32_t j0 = 0; j0 < n; j0 += 32u) {
    const uint32_t d = bm + j0 + lane;
    uint32_t code1 = DEC_DIES;
    if (j0 + lane < n) {
      const uint32_t g = ps.moved[warp][j0 + lane];
      Rec a;
      load_cols<CS>(w.src, g, a);
      const uint32_t female = (__ldg(w.src.flags + g) >> 3) & 1u;
      implied_fields<RG, WIDE>(a);
      a.female = female;
      (void)update_agent<true, false, true, true, !WIDE>(w.c, mc.kill, RG, g, a, acc, DEC_MOVES);
      if (RG == EGG || RG == BMD) {  // the owed normal draw (include/gpuRand.h:56-63)
        if (a.bm == BM_LARVA_DELAY) a.delay = __uint_as_float(finish_box_muller(w.c, mc, g, BM_LARVA_DELAY, 0u));
        else if (a.bm == BM_EGG_BATCH) a.avail = finish_box_muller(w.c, mc, g, BM_EGG_BATCH, a.batches);
      }
      store_cols<CM>(w.dst, d, a);
      if (RG >= PUPA && female) {  // statistics of the next pool (kernel/calcGender.cl:24-37)
        fem += 1u;
        inf += a.sporo >= 1.0f ? 1u : 0u;
      }
      if (AHEAD) code1 = decide<NX, WIDE>(w.c1, mc.kill, d, a, da);
      put(w.dst.flags + d, NX | (female << 3) | (code1 << 4));
    }
    if (AHEAD) add_tally<NX>(w, t, bm + j0, min(n - j0, 32u), d, tally_count(code1));
  }
  if (AHEAD) {
    flush_tally<NX>(w, t);
    add_decided<NX, NX>(da, sum);
  }
  if (RG >= PUPA) add_moved<RG>(fem, inf, acc, sum);
  return bm + n;
}

// The update/scatter pass over slots [lo, hi) of range RG. base (lanes 0-7):
// the next slot of next state `lane` for this warp's survivors; returned past
// the range's. A survivor's slot is that plus its rank among the survivors
// of its state in the row (two ballots: an agent stays or moves on to one
// other state). The survivors of a state are consecutive, so the stores of a
// row coalesce.
// AHEAD: each survivor's decision of the step after is taken here as well,
// while its record is in registers: its slot in the next pool, that step's
// inputs and (from this step's decisions) that pool's L1de and size are all
// known. The decisions go into the flags, their counts to the next pool's
// spans and supers, and no count pass is needed before the next step.
template <bool B>
struct Flag { static constexpr bool value = B; };
template <int I, bool WIDE, bool AHEAD, int RG>
__device__ __noinline__ uint32_t scatter_range(uint32_t lo, uint32_t hi, uint32_t base) {
  constexpr int NX = next_state(RG);
  constexpr uint32_t CS = state_cols(RG, WIDE);
  using RING = Ring<CS, WIDE ? 2 : 1, I>;
  constexpr uint32_t ROWS = RING::kSlots / 32;
  static_assert(RING::kSlots + 31 < kMoved && RING::kSlots <= kSpanMin, "a chunk's moves fit behind the ones that wait; a chunk fills at most two spans");
  PassShared& ps = pass_shared();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = lanemask_lt();
  const WarpRep& w = ps.rep[warp];
  const ModelConst& mc = ps.mc;
  uint32_t* const moved = ps.moved[warp];
  WarpSum& sum = ps.sum[warp];
  uint32_t bs = __shfl_sync(0xffffffffu, base, RG), bm = __shfl_sync(0xffffffffu, base, NX);
  const uint32_t es = w.next.r[RG].end, span = hi - lo;
  Tally ts = {0, 0, 0};
  DecideAcc da;
  clear_acc(da);
  uint32_t bad = 0, qn = 0;  // qn: slots that wait to be moved on
  // the rows' moves (mm: a row's lanes; g: the lane's slot) into the queue, and out of it
  auto queue_moves = [&](uint32_t mm, uint32_t g) {
    if ((mm >> lane) & 1u) moved[qn + __popc(mm & lt)] = g;
    qn += __popc(mm);
  };
  auto move_waiting = [&](bool last) {
    if (qn >= (last ? 1u : 32u)) {
      const uint32_t n = last ? qn : qn & ~31u;
      __syncwarp();
      bm = move_on<WIDE, AHEAD, RG>(n, bm);
      qn -= n;
      __syncwarp();
      const uint32_t rest = lane < qn ? moved[n + lane] : 0u;
      __syncwarp();
      if (lane < qn) moved[lane] = rest;
    }
  };
  if constexpr (AHEAD && !WIDE && RG <= LARVA) {
    // Eggs and larvae that stay: nearly all of every pool. The same update
    // and decision as update_agent's, laid out without branches (every lane
    // computes, the survivors store), a chunk's bookkeeping done once. What
    // bounds it is the instructions of a row (about 45 and 70).
    const DevPool src = w.src, dst = w.dst;
    const uint32_t h13 = w.c1.rng_c13[0], hz2 = w.c1.rng_z2[0], hk4 = w.c1.rng_k4[0], hkill = mc.kill.aquatic;
    const float hdev = w.c.larvaDev, hdev1 = w.c1.larvaDev;
    const bool htt = w.c1.tt & (RG == EGG ? TT_EGG : TT_LARVA), hcide = RG == LARVA && w.c1.env.larvacideValue > 0.0f;
    uint32_t youngest = 0xffffffffu, oldest = 0, hatched = 0, seen = 0;
    stream_range<RING, CS>(ps.ring[warp], src, src.flags, nullptr, lo, hi, [&](const uint8_t* st, uint32_t g0) {
      const uint8_t* const stf = st + RING::kByteOffset + lane;
      const bool whole = g0 >= lo && hi - g0 >= RING::kSlots;
      auto code_of = [&](uint32_t k) {
        const uint32_t code = stf[32 * k] & 0x30u;
        return whole || g0 + 32u * k + lane - lo < span ? code : 0u;
      };
      uint32_t ms[ROWS], n = 0, any = 0;
#pragma unroll
      for (uint32_t k = 0; k < ROWS; k++) {
        const uint32_t code = code_of(k);
        ms[k] = __ballot_sync(0xffffffffu, code == DEC_STAYS << 4);
        any |= code;
        n += __popc(ms[k]);
      }
      if (bs + n > es) {  // no store leaves the state's run
        bad = SAMPO_DEV_ERR_TILECOUNT;
        return;
      }
      if (bs >= ts.end) {
        hatched += ts.cnt >> 16;
        next_tally<RG>(w, ts, bs);
      }
      seen |= n;
      auto rows = [&](auto crosses) {  // crosses: the chunk's survivors reach past the span's end
        uint32_t past = 0;
#pragma unroll
        for (uint32_t k = 0; k < ROWS; k++) {
          const uint32_t fl = stf[32 * k];
          const float* f = reinterpret_cast<const float*>(st) + 32u * k + lane;
          const float delay = f[RING::offset(C_DELAY) / 4], age = f[RING::offset(C_AGE) / 4] + 1.0f;
          const float cld = RG == LARVA ? f[RING::offset(C_UNI) / 4] + hdev : 0.0f;
          const uint32_t d = bs + __popc(ms[k] & lt);
          const bool live = (ms[k] >> lane) & 1u;
          bs += __popc(ms[k]);
          // the step after: mortality, then the transition (update_agent<false>)
          uint32_t kill = hkill;
          float q = 0.0f;
          if (RG == LARVA) {
            q = whole_age_quotient(live ? age : 24.0f);
            const uint32_t days = whole_days(q);
            kill = w.larvaKill1[days < 99u ? days : 99u];
            if (live && kill == 0u) da.acc.bad = 1u;
          }
          bool lives = live && rng_bits(h13, hz2, hk4, d) >= kill;
          if (RG == LARVA && hcide) lives = lives && !(age - 23.0f == 1.0f && rng(w.c1, 2, d) <= w.c1.env.larvacideValue);
          const bool due = htt && (RG == EGG ? age + 1.0f >= delay : cld + hdev1 >= delay);
          const uint32_t c = lives ? (due ? 1u << 16 : 1u) : 0u;
          ts.cnt += c;
          if (crosses.value && d >= ts.end) past += c;
          if (RG == LARVA && lives && !due) {  // its whole days an hour on
            const uint32_t days = whole_days_next(q);
            da.l1 += days;
            youngest = min(youngest, days);
            oldest = max(oldest, days);
          }
          put_if<RG>(live, dst, d, age, delay, cld, (fl & 8u) | (lives ? (due ? RG | DEC_MOVES << 4 : RG | DEC_STAYS << 4) : (uint32_t)RG));
        }
        if (crosses.value) {
          ts.cnt -= past;
          hatched += ts.cnt >> 16;
          next_tally<RG>(w, ts, ts.end);
          ts.cnt = past;
        }
      };
      if (bs + n > ts.end) rows(Flag<true>{});
      else rows(Flag<false>{});
      if (__any_sync(0xffffffffu, any & (DEC_MOVES << 4))) {
#pragma unroll 1
        for (uint32_t k = 0; k < ROWS; k++) queue_moves(__ballot_sync(0xffffffffu, code_of(k) == DEC_MOVES << 4), g0 + 32u * k + lane);
      }
      move_waiting(hi - g0 <= RING::kSlots);
    });
    hatched += ts.cnt >> 16;
    if (RG == EGG) {  // hatched: 24 hours old
      da.l1 = hatched;
      if (hatched) da.dmin = da.dmax = 1u;
    } else {
      da.devoob = seen ? w.c1.devOOB : 0u;
      if (youngest != 0xffffffffu) {  // (a loaded larva may be in its day 0)
        da.dmin = min(youngest, 99u);
        da.dmax = min(oldest, 99u);
      }
    }
  } else {
    const DevPool &src = w.src, &dst = w.dst;
    const uint8_t* const dec = WIDE ? w.dec : nullptr;
    Acc acc = {0, 0, 0, 0, 0, 0};
    uint32_t fem = 0, inf = 0;
    stream_range<RING, CS>(ps.ring[warp], src, src.flags, dec, lo, hi, [&](const uint8_t* st, uint32_t g0) {
#pragma unroll kRowUnroll
      for (uint32_t k = 0; k < ROWS; k++) {
        const uint32_t i = 32u * k + lane, g = g0 + i;
        const uint32_t fl = st[RING::kByteOffset + i];
        uint32_t code = WIDE && dec ? st[RING::kByteOffset + RING::kSlots + i] : (fl >> 4) & 3u;
        if (g - lo >= span) code = DEC_DIES;
        uint32_t ms = __ballot_sync(0xffffffffu, code == DEC_STAYS);
        const uint32_t mm = __ballot_sync(0xffffffffu, code == DEC_MOVES);
        uint32_t n = __popc(ms);
        if (bs + n > es) {  // no store leaves the state's run
          bad = SAMPO_DEV_ERR_TILECOUNT;
          ms = n = 0;
        }
        const uint32_t d = bs + __popc(ms & lt);
        uint32_t code1 = DEC_DIES;
        if ((ms >> lane) & 1u) {
          Rec a;
          read_chunk<RING, CS>(st, i, a);
          implied_fields<RG, WIDE>(a);
          a.female = (fl >> 3) & 1u;
          (void)update_agent<true, false, true, true, !WIDE>(w.c, mc.kill, RG, g, a, acc, DEC_STAYS);
          store_cols<CS>(dst, d, a);
          if (RG >= IMMATURE && a.female) {  // statistics of the next pool (kernel/calcGender.cl:24-37)
            fem += 1u;
            inf += a.sporo >= 1.0f ? 1u : 0u;
          }
          if (AHEAD) code1 = decide<RG, WIDE>(w.c1, mc.kill, d, a, da);
          put(dst.flags + d, RG | (fl & 8u) | (code1 << 4));  // (the range's state: a loaded pool's state bits may differ)
        }
        if (AHEAD) add_tally<RG>(w, ts, bs, n, d, tally_count(code1));
        bs += n;
        if (mm) queue_moves(mm, g);
        if (RG == GRAVID && code == DEC_TRAPPED) {  // her last hour counts (kernel/updateAgents.cl:247-255)
          acc.cycles += 1u;
          acc.sumCycles += reinterpret_cast<const uint32_t*>(st)[RING::offset(C_CYCLE) / 4 + i] + 1u;
        }
      }
      move_waiting(hi - g0 <= RING::kSlots);
    });
    if (RG >= IMMATURE) add_moved<RG>(fem, inf, acc, sum);
  }
  if (AHEAD) {
    if (ts.end) flush_tally<RG>(w, ts);
    add_decided<RG, RG>(da, sum);
  }
  if (bad && lane == 0) sum.error |= bad;
  return lane == (uint32_t)RG ? bs : lane == (uint32_t)NX ? bm : base;
}

template <int I, bool WIDE, bool AHEAD>
struct ScatterRanges {
  uint32_t& base;
  template <int RG>
  __device__ __forceinline__ void operator()(uint32_t lo, uint32_t hi) {
    base = scatter_range<I, WIDE, AHEAD, RG>(lo, hi, base);
  }
};

// The update/scatter pass: units 0 .. nspans-1 of a replicate are its spans,
// the rest its new eggs. A span's first slot in every next-state range comes
// from the decisions' counts: its super's prefix plus the spans before it in
// the super (one 16-byte word per lane). No warp waits for another.
template <int I, bool WIDE, bool AHEAD>
__global__ void __launch_bounds__(kBlock, 3) k_scatter(KParams p) {
  PassShared& ps = pass_shared();
  uint32_t* s_pre = reinterpret_cast<uint32_t*>(pass_shared_memory + sizeof(PassShared));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  load_model_const(p.mc, ps.mc);
  wait_previous_kernel();
  const uint32_t min_span = p.bat->minSpan;
  plan_tickets(p.nrep, s_pre, ps.scan, [&](uint32_t r) -> uint32_t {
    SimDev* sim = p.reps[r].sim;
    if (!sim->active) return 0u;
    uint32_t cnt[8];
    for (int k = 0; k < 8; k++) cnt[k] = sim->cnt[k];
    const uint32_t ne = sim->dec.newEggs;
    if (!layout_fits(cnt, ne, sim->capacity)) {
      if (blockIdx.x == 0) atomicOr(&sim->error, SAMPO_DEV_ERR_CAPACITY);
      return 0u;
    }
    const uint32_t end = sim->pop.r[GRAVID].end;
    const uint32_t span = span_size(end, min_span);
    return units_of(end, span) + units_of(ne, span);
  });
  __syncthreads();
  const uint32_t total = s_pre[p.nrep], stride = gridDim.x * kWarps;
  WarpRep& w = ps.rep[warp];
  uint32_t cur_rep = kNoRep;
  WarpSum& sum = ps.sum[warp];
  if (lane == 0) clear_sum(sum);
  // lane 0, before this warp's sums go into its replicate's
  auto end_rep = [&]() {
    if (AHEAD && cur_rep != kNoRep && !w.ahead) {  // (its decisions were taken for nothing)
      sum.dec = Decided{0u, 0u, 0xffffffffu, 0u};
      sum.error &= SAMPO_DEV_ERR_TILECOUNT;
    }
  };
  for (uint32_t t = blockIdx.x * kWarps + warp; t < total; t += stride) {
    const uint32_t r = find_rep(s_pre, p.nrep, t);
    if (r != cur_rep) {  // uniform
      if (cur_rep != kNoRep && lane == 0) {
        end_rep();
        flush_sum(sum, p.reps[cur_rep].sim, &p.reps[cur_rep].sim->ahead_dec);
      }
      load_warp_rep<true, AHEAD>(p.reps[r], min_span, w);
      cur_rep = r;
    }
    const uint32_t sp = t - s_pre[r];
    if (AHEAD) {  // this unit's share of the span counts that the pass after the next adds to
      const uint32_t z1 = min((sp + 1u) * w.clearPer, w.clear);
      for (uint32_t z = sp * w.clearPer + lane; z < z1; z += 32u) w.spans2[z] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (sp < w.nspans) {
      const uint32_t i = (sp & ~31u) + lane;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (i <= sp) v = __ldg(w.spans + i);
      const uint32_t pre = lane < 8 ? __ldg(w.superPre + (size_t)(sp >> 5) * 8 + lane) : 0u;
      uint4 own, before;
      own.x = __shfl_sync(0xffffffffu, v.x, sp & 31u);
      own.y = __shfl_sync(0xffffffffu, v.y, sp & 31u);
      own.z = __shfl_sync(0xffffffffu, v.z, sp & 31u);
      own.w = __shfl_sync(0xffffffffu, v.w, sp & 31u);
      before.x = __reduce_add_sync(0xffffffffu, v.x) - own.x;
      before.y = __reduce_add_sync(0xffffffffu, v.y) - own.y;
      before.z = __reduce_add_sync(0xffffffffu, v.z) - own.z;
      before.w = __reduce_add_sync(0xffffffffu, v.w) - own.w;
      const uint32_t b = lane & 7;
      const uint32_t base0 = (b == EGG ? w.newEggs : w.next.r[b].start) + pre + state_count(before, b);
      uint32_t base = base0;
      const uint32_t end = w.pop.r[GRAVID].end, u0 = sp * w.span;
      const uint32_t u1 = end - u0 > w.span ? u0 + w.span : end;
      for_ranges(w.pop, u0, u1, ScatterRanges<I, WIDE, AHEAD>{base});
      // the decisions and their counts must agree on the span's survivors
      const bool differ = __any_sync(0xffffffffu, lane < 8 && base - base0 != state_count(own, b));
      if (differ && lane == 0) sum.error |= SAMPO_DEV_ERR_TILECOUNT;
    } else {
      // ---- new eggs at [0, newEggs) of the next buffer ----
      const uint32_t e0 = (sp - w.nspans) * w.span, ne = w.newEggs;
      const uint32_t e1 = ne - e0 > w.span ? e0 + w.span : ne;
      const DevPool dst = w.dst;
      constexpr bool ahead = AHEAD;
      Tally ts = {0, 0, 0};
      DecideAcc da;
      clear_acc(da);
      for (uint32_t r0 = e0; r0 < e1; r0 += 32u) {
        const uint32_t id = r0 + lane;
        const bool in = id < e1;
        uint32_t code1 = DEC_DIES;
        if (in) {
          Rec a;
          new_egg(w.c, id, a);
          store_cols<state_cols(EGG, WIDE)>(dst, id, a);
          const uint32_t female = a.female;
          if (ahead) code1 = decide<EGG, WIDE>(w.c1, ps.mc.kill, id, a, da);
          put(dst.flags + id, EGG | (female << 3) | (code1 << 4));
        }
        if (ahead) add_tally<EGG>(w, ts, r0, min(e1 - r0, 32u), id, tally_count(code1));
      }
      if (ahead) {
        flush_tally<EGG>(w, ts);
        add_decided<EGG, EGG>(da, sum);
      }
    }
  }
  if (lane == 0) {
    end_rep();
    sum.rep = cur_rep;
    sum.spans = 0;
  }
  (void)flush_sums(p.reps, ps.sum, true);
}

// ------------------------------------------------------------------------
// Initial population of p.reps[0]: initAgents over [0, n)
// (kernel/initAgents.cl:26-65), optionally with ages 24*U{0..age_days_max}
// from splitmix64 (an extension).
// ------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

__global__ void k_init_eggs(KParams p, uint32_t n, float T0, const sampo_seeds* seeds, int age_days_max, uint64_t age_seed, int full) {
  __shared__ StepCtx c;
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; k++) {
      c.rng_c13[k] = taus_step(seeds[k].z1 + 128u, 13, 19, 12, 4294967294u) ^ taus_step(seeds[k].z3 + 128u, 3, 11, 17, 4294967280u);
      c.rng_z2[k] = seeds[k].z2 + 128u;
      c.rng_k4[k] = 1664525u * seeds[k].z4;
    }
    species_step(T0, 0u, c);  // eggsIncubation(temperature[0]) (kernel/initAgents.cl:57)
  }
  __syncthreads();
  const DevPool dst = p.reps[0].pool[0];
  // 64-bit counters: a bound within one grid stride of 2^32 must not wrap
  for (uint64_t i64 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i64 < n; i64 += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t id = (uint32_t)i64;
    Rec a;
    new_egg(c, id, a);
    if (age_days_max >= 0) {
      uint64_t z = mix64(age_seed ^ mix64((uint64_t)id));
      float h = 24.0f * (float)(uint32_t)((z >> 32) % ((uint64_t)age_days_max + 1));
      a.age = h; a.his = h;
    }
    if (full) store_cols<C_ALL>(dst, id, a);
    else store_cols<state_cols(EGG, false)>(dst, id, a);
    dst.flags[id] = (uint8_t)(EGG | (a.female << 3));
  }
}

// Before and after a timing trial of the step kernels: zero what they add to
// (eggs laid, next-pool statistics) and the survivor counts. Their other
// writes - the next buffer, and decisions and span counts equal to the ones
// the real step computes - leave the simulation's course unchanged.
__global__ void k_trial_reset(KParams p) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < p.nrep; r += gridDim.x * blockDim.x) {
    SimDev* sim = p.reps[r].sim;
    for (int k = 0; k < 8; k++) sim->cnt[k] = 0;
    sim->dec = Decided{0u, 0u, 0xffffffffu, 0u};
    sim->acc_fem = sim->acc_inf = 0;
    for (int k = 0; k < 4; k++) sim->acc_bnc[k] = 0;
  }
}

// The columns a narrow record implies (state_cols), written out, the decision
// bits taken out of the flags, and zeros into the slots between the ranges,
// for every replicate of p: what a reader of the pool's columns expects.
__global__ void k_widen(KParams p) {
  for (uint32_t r = 0; r < p.nrep; r++) {
    const SimDev* sim = p.reps[r].sim;
    const sampo_population pop = sim->pop;
    const DevPool d = p.reps[r].pool[sim->cur];
    if (!d.age) continue;  // an empty slot of a batch
    const uint32_t end = pop.r[GRAVID].end;
    for (uint64_t g64 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g64 < end; g64 += (uint64_t)gridDim.x * blockDim.x) {
      const uint32_t g = (uint32_t)g64;
      const int rg = range_of(pop, g);
      if (rg < 0) {  // a slot between two ranges
        store_cols<C_ALL>(d, g, Rec{});
        d.flags[g] = 0;
        continue;
      }
      d.flags[g] &= 15u;
      if (p.wide || rg >= BMS) continue;
      if (rg == EGG) { d.his[g] = d.age[g]; d.uni[g] = 0u; }
      if (rg == LARVA) d.his[g] = d.age[g] - 24.0f;
      d.sporo[g] = 0.0f; d.avail[g] = 0u; d.cycle[g] = 0u; d.hbc[g] = 0u; d.batches[g] = 0u;
    }
  }
}

// Whether an agent's record holds anything its state does not imply (see
// state_cols), or an age that is not a whole number of hours below 2^20 (the
// narrow passes take days from whole hours, and a larva's hoursInState from
// its age; no agent lives another 2^20 hours).
__device__ __forceinline__ bool wide_record(const DevPool& s, uint32_t g, int rg) {
  const float age = s.age[g], his = s.his[g];
  if (!(age >= 0.0f && age < 1048576.0f) || age != floorf(age)) return true;
  if (rg >= BMS) return false;
  bool w = __float_as_uint(s.sporo[g]) != 0u || s.avail[g] || s.cycle[g] || s.hbc[g] || s.batches[g];
  if (rg == EGG) w |= __float_as_uint(his) != __float_as_uint(age) || s.uni[g];
  if (rg == LARVA) w |= __float_as_uint(his) != __float_as_uint(age - 24.0f);
  return w;
}

// Statistics of p.reps[0]'s current pool, accumulated into acc_*; PS_CHECK:
// also whether its records are wide, PS_CLEAR: also clears the supers,
// PS_ROWS: the records and state of the one-launch step's rows. Only
// the ranges that the statistics come from are read (larvae and adults; with
// PS_CHECK all), as one sequence of four-slot groups (16-byte loads), so that
// a thread has few turns of a load latency each; a loop over all slots that
// looked its range up, and an add per warp to the same words, took 32 us at
// 5e6 agents where this takes 14.
__global__ void __launch_bounds__(256) k_pool_stats(KParams p, uint32_t flags) {
  __shared__ WarpSum sums[kWarps];
  const RepParams& rp = p.reps[0];
  SimDev* sim = rp.sim;
  const sampo_population pop = sim->pop;
  const DevPool src = rp.pool[sim->cur];
  const bool check = flags & PS_CHECK;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  uint32_t l1 = 0, fem = 0, inf = 0, dmin = 0xffffffffu, dmax = 0;
  bool wide = false;
  if (flags & PS_CLEAR) {
    const uint32_t n = units_of(span_count(pop.r[GRAVID].end, 0), 32);
    for (uint32_t i = tid; i < n; i += threads) rp.supers[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (flags & PS_ROWS) {
    const uint32_t n = (uint32_t)small_group_words(rp.smallTiles) / 4u;
    uint4* const groups = reinterpret_cast<uint4*>(rp.smallRows);
    for (uint32_t i = tid; i <= n; i += threads) groups[i < n ? i : n + rp.smallTiles] = make_uint4(0u, 0u, 0u, 0u);  // (the state lies behind the tiles)
  }
  uint32_t upto[8], groups = 0;  // groups of the ranges up to each
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const bool read = (check || k == LARVA || k >= IMMATURE) && pop.r[k].end > pop.r[k].start;
    groups += read ? (pop.r[k].end - (pop.r[k].start & ~3u) + 3u) / 4u : 0u;
    upto[k] = groups;
  }
#pragma unroll 2
  for (uint32_t q = tid; q < groups; q += threads) {
    int rg = 0;
    uint32_t before = 0, lo = pop.r[0].start, hi = pop.r[0].end;
#pragma unroll
    for (int k = 1; k < 8; k++)
      if (q >= upto[k - 1]) {
        rg = k;
        before = upto[k - 1];
        lo = pop.r[k].start;
        hi = pop.r[k].end;
      }
    const uint32_t g = (lo & ~3u) + 4u * (q - before);
    if (check)
      for (uint32_t i = max(g, lo); i < min(g + 4u, hi); i++) wide |= wide_record(src, i, rg);
    if (rg == LARVA) {
      const float4 v = *reinterpret_cast<const float4*>(src.age + g);
      const float age[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        if (g + i < lo || g + i >= hi) continue;
        const uint32_t dd = age_days(age[i]);
        l1 += age_days_uncapped(age[i]);
        dmin = min(dmin, dd);
        dmax = max(dmax, dd);
      }
    } else if (rg >= IMMATURE) {
      const uint32_t fl = *reinterpret_cast<const uint32_t*>(src.flags + g);
      const float4 v = *reinterpret_cast<const float4*>(src.sporo + g);
      const float sporo[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        const uint32_t female = g + i >= lo && g + i < hi ? (fl >> (8 * i + 3)) & 1u : 0u;
        fem += female;
        inf += sporo[i] >= 1.0f ? female : 0u;
      }
    }
  }
  wide = __any_sync(0xffffffffu, wide);
  l1 = __reduce_add_sync(0xffffffffu, l1);
  fem = __reduce_add_sync(0xffffffffu, fem);
  inf = __reduce_add_sync(0xffffffffu, inf);
  dmin = __reduce_min_sync(0xffffffffu, dmin);
  dmax = __reduce_max_sync(0xffffffffu, dmax);
  // one add per CTA and word
  if ((threadIdx.x & 31) == 0) {
    WarpSum& t = sums[threadIdx.x >> 5];
    clear_sum(t);
    t.dec.L1de = l1;
    t.dec.dmin = dmin;
    t.dec.dmax = dmax;
    t.fem = fem;
    t.inf = inf;
    t.rep = t.spans = 0;
    if (wide) sim->wide = 1u;
  }
  (void)flush_sums(p.reps, sums, false);
}

// ageHistogram (kernel/ageHistogram.cl:13-35) of p.reps[0] with
// warp-aggregated shared atomics: lanes that fall in the same bin add once.
__global__ void k_histogram(KParams p, uint32_t* hist) {
  __shared__ uint32_t h[100];
  for (int k = threadIdx.x; k < 100; k += blockDim.x) h[k] = 0;
  __syncthreads();
  SimDev* sim = p.reps[0].sim;
  const sampo_population pop = sim->pop;
  const DevPool src = p.reps[0].pool[sim->cur];
  const uint32_t lo = pop.r[IMMATURE].start, hi = pop.r[GRAVID].end;
  const uint32_t span = hi > lo ? hi - lo : 0u;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < span; base += stride) {  // warp-uniform
    const uint32_t g = lo + (uint32_t)base + threadIdx.x;
    int rg = (base + threadIdx.x < span) ? range_of(pop, g) : -1;
    uint32_t bin = 0xffffffffu;
    if (rg >= IMMATURE) {
      bin = age_days_uncapped(src.age[g]);
      bin = bin < 99u ? bin : 99u;
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, bin);
    if (bin != 0xffffffffu && (threadIdx.x & 31) == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&h[bin], (uint32_t)__popc(peers));
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 100; k += blockDim.x)
    if (h[k]) atomicAdd(&hist[k], h[k]);
}

// Diagnostic: the model's transcendental definitions evaluated on the device.
__global__ void k_eval_math(int fn, const float* x, const float* y, float* out, uint32_t n) {
  for (uint64_t i64 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i64 < n; i64 += (uint64_t)gridDim.x * blockDim.x) {
    const size_t i = (size_t)i64;
    float v = 0.0f;
    switch (fn) {
      case 0: v = sampo_expf(x[i]); break;
      case 1: v = sampo_logf(x[i]); break;
      case 2: v = sampo_sinf(x[i]); break;
      case 3: v = sampo_powf(x[i], y[i]); break;
      case 4: v = sampo_logf_bm(x[i]); break;
      case 5: v = sampo_sinf_bm(x[i]); break;
      default: break;
    }
    out[i] = v;
  }
}

}  // namespace sampo
