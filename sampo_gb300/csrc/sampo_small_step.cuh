// sampo_small_step.cuh - the hourly step of one simulation in one launch, for
// pools of up to a few hundred 1024-slot tiles (sm_103a).
//
// At that size the three-kernel step (k_count, k_scatter, k_publish) is bound
// by each kernel's start-up and latency chain, not by bandwidth. k_step_small
// does the same step in one cooperative launch with one CTA per tile:
//
//  phase 1  CTA b loads tile b (TMA bulk copies) and runs the full update of
//           its agents once (killAgents + updateAgents with the species
//           functions and the normal draws). The updated records stay in the
//           CTA's shared memory with their next state in the flag byte; the
//           CTA builds the tile's prefix table over its (round, warp) chunks
//           in shared memory and publishes the tile's survivors per next
//           state, its eggs laid and its share of the next pool's statistics
//           (calcL1de.cl, calcGender.cl) to global memory.
//  barrier  a grid barrier with a bounded wait.
//  phase 2  every CTA sums the counts (SmallRows): the totals give the next
//           layout (kernel/oldToNewAgents.cl:57-95), the tiles before its own
//           the tile's first slot in each next-state range. It writes its
//           survivors from shared memory to their slots in the next buffer
//           and the new eggs of its egg tiles at [0, newEggs)
//           (kernel/initAgents.cl:26-65), then computes the next step's
//           state from the totals (the k_publish code); the last CTA also
//           stores it for the host.
//  barrier  a second grid barrier; the next hour's tile copies go out.
//
// Pools with more tiles than CTAs are still stepped correctly: CTA b also
// takes tiles b + G, b + 2G, ... (G CTAs); their decisions are counted in
// phase 1 and the tile is loaded and updated again in phase 2.
//
// A narrow pool's records are read and written by the columns of their state
// (state_cols), as in the other passes (a year from 1e4 eggs: 11.9 us an hour
// with whole records, 11.0 so).
// A species compiled at run time has it too (20,000 eggs for a month: 21.7 ms
// with three kernels an hour, 13.2 ms with one launch a day).
#pragma once
#include "sampo_step_kernels.cuh"

namespace sampo {

constexpr int kSmallThreads = kBlock;      // eight warps, I slots per thread (tiles of kBlock * I slots: I = 1, 2 or 4)
constexpr int kSmallMinBlocks = 3;         // resident CTAs per SM the registers are sized for
__host__ __device__ constexpr uint32_t small_stage(int items) { return 9 * kBlock * items * 4 + kBlock * items; }  // ten columns
constexpr uint32_t kSmallRows = 9;         // per-tile counts: survivors by next state, eggs laid
constexpr uint8_t kGone = 0xffu;           // flag byte of a slot without a survivor
constexpr uint32_t kSmallHours = 24;       // most hours of a launch, whose constants a CTA holds in shared memory
// Per-CTA statistics of the next pool (CTA b's column, b < the tiles):
// L1de, females, infective, cycles, sum of cycles, bites, infective bites
// (sums) and the min and max larva age in days.
enum : uint32_t { SA_L1 = 0, SA_FEM, SA_INF, SA_CYC, SA_SUMCYC, SA_BITES, SA_IBITES, SA_DMIN, SA_DMAX, kSmallStats };
static_assert(kSmallRows == 9 && SA_DMIN == 7 && kSmallStats == SA_DMAX + 1 && kSmallStats == 9, "a group's record, by fours");
// The sizes of a kernel built for I slots per thread. A tile's prefix table
// has, for each (round, warp) chunk of 32 slots (slot k * kBlock + tid is
// round k of warp tid / 32) and for the whole tile, the survivors of the
// chunks before it by next state (16-bit pairs) and over all states.
constexpr uint32_t kPreEntryWords = 5;
#define SAMPO_TILE_CONSTANTS(I)                    \
  constexpr int kItems = (I);                      \
  constexpr int kTile = kBlock * (I);              \
  constexpr uint32_t kChunks = (uint32_t)(I) * kWarps; \
  constexpr uint32_t kColBytes = (uint32_t)kTile * 4;  \
  static_assert(kChunks <= 32, "one chunk per lane");  \
  (void)kItems; (void)kChunks; (void)kColBytes

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A grid barrier in two halves. small_grid_arrive (every thread): the CTA's
// writes so far are ordered before its arrival by the CTA barrier and the
// release of the arrival. small_grid_wait (every thread): all CTAs of the
// grid (co-resident: a cooperative launch) wait until the arrival counter
// reaches `target` (the grid size times the barriers passed so far in the
// launch); the acquire of the counter orders the reads that follow. Bounded:
// false when the others did not arrive within the limit; every thread gets
// the same answer. Work that needs no other CTA can go between the halves.
__device__ __forceinline__ void small_grid_arrive(uint32_t* bar) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ bool small_grid_wait(uint32_t* bar, uint32_t target, uint32_t* s_flag) {
  if (threadIdx.x == 0) {
    uint32_t ok = 0;
    for (uint32_t i = 0; i < kWaitLimit; i++) {
      if (ld_acquire_u32(bar) >= target) { ok = 1; break; }
      if (i >= 32) __nanosleep(32);
    }
    *s_flag = ok;
  }
  __syncthreads();
  return *s_flag != 0;
}
__device__ bool small_grid_barrier(uint32_t* bar, uint32_t target, uint32_t* s_flag) {
  small_grid_arrive(bar);
  return small_grid_wait(bar, target, s_flag);
}

struct SmallAcc {
  Acc acc;                            // counters of the update (bites, cycles, eggs laid, table misses)
  uint32_t l1, fem, inf, dmin, dmax;  // statistics of the next pool
  uint32_t devoob, tilebad;
};

// Phase 1 (and phase 2 for a tile updated again): the full update of the
// tile in stage memory st (slots lo .. lo + kTile of the current pool). With
// KEEP the updated records and their next state (flag byte; kGone for none)
// are written back to the stage. Every (round, warp) chunk's survivors by
// next state go to s_ent. EGGS / STATS: the eggs laid / the update's
// counters and the next pool's statistics go to sa (a tile updated twice
// counts its eggs the first time and the rest the second).
template <int I, bool KEEP, bool EGGS, bool STATS>
__device__ __forceinline__ void small_update_tile(const StepCtx& c, const ModelConst& mc, const sampo_population& pop,
                                                  bool whole, uint8_t* st, uint32_t lo, uint32_t end, uint2* s_ent, SmallAcc& sa) {
  SAMPO_TILE_CONSTANTS(I);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* c_age = (float*)(st + 0 * kColBytes);
  float* c_his = (float*)(st + 1 * kColBytes);
  float* c_delay = (float*)(st + 2 * kColBytes);
  float* c_sporo = (float*)(st + 3 * kColBytes);
  uint32_t* c_uni = (uint32_t*)(st + 4 * kColBytes);
  uint32_t* c_avail = (uint32_t*)(st + 5 * kColBytes);
  uint32_t* c_cycle = (uint32_t*)(st + 6 * kColBytes);
  uint32_t* c_hbc = (uint32_t*)(st + 7 * kColBytes);
  uint32_t* c_batches = (uint32_t*)(st + 8 * kColBytes);
  uint8_t* c_flags = st + 9 * kColBytes;
  Acc t = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
  for (int k = 0; k < kItems; k++) {
    const uint32_t i = k * kBlock + tid;
    const uint32_t g = lo + i;
    const int rg = g < end ? range_of(pop, g) : -1;
    uint32_t pk0 = 0, pk1 = 0;  // this slot's next state as an 8-bit counter: states 0-3, 4-7
    uint8_t fb = kGone;
    if (rg >= 0) {
      Rec a;
      // (state_cols: what a narrow record's state implies is not there)
      a.age = c_age[i]; a.delay = c_delay[i];
      a.uni = !whole || rg != EGG ? c_uni[i] : 0u;
      a.his = !whole || rg >= PUPA ? c_his[i] : rg == EGG ? a.age : a.age - 24.0f;
      a.sporo = 0.0f; a.avail = a.cycle = a.hbc = a.batches = 0u;
      if (!whole || rg >= BMS) {
        a.sporo = c_sporo[i]; a.avail = c_avail[i]; a.cycle = c_cycle[i]; a.hbc = c_hbc[i]; a.batches = c_batches[i];
      }
      a.female = (c_flags[i] >> 3) & 1u;
      a.bm = BM_NONE;
      sa.devoob |= (rg == LARVA) & c.devOOB;
      // (days from whole hours without the division: a uniform choice)
      const uint32_t days = rg != LARVA && rg < IMMATURE ? 0u : whole ? age_days<true>(a.age) : age_days(a.age);
      const int ns = update_agent<true, true, false, false, false, true>(c, mc.kill, rg, g, a, t, DEC_STAYS, days);
      if (ns >= 0) {
        if (a.bm != BM_NONE) {  // the owed normal draw (include/gpuRand.h:56-63)
          const uint32_t v = finish_box_muller(c, mc, g, a.bm, a.batches);
          if (a.bm == BM_LARVA_DELAY) a.delay = __uint_as_float(v);
          else a.avail = v;
        }
        if (ns < 4) pk0 = 1u << (8 * ns);
        else pk1 = 1u << (8 * (ns - 4));
        fb = (uint8_t)(ns | (a.female << 3));
        if (STATS) {  // kernel/calcL1de.cl:28-30, kernel/calcGender.cl:24-37
          if (ns == LARVA) {
            const uint32_t du = whole ? whole_age_days(a.age) : age_days_uncapped(a.age);
            const uint32_t dd = whole ? min(du, 99u) : age_days(a.age);
            sa.l1 += du;
            sa.dmin = min(sa.dmin, dd); sa.dmax = max(sa.dmax, dd);
          } else if (ns >= IMMATURE && a.female) {
            sa.fem += 1u;
            sa.inf += a.sporo >= 1.0f ? 1u : 0u;
          }
        }
        if (KEEP) {
          c_age[i] = a.age; c_delay[i] = a.delay;
          if (!whole || ns != EGG) c_uni[i] = a.uni;
          if (!whole || ns >= PUPA) c_his[i] = a.his;
          if (!whole || ns >= BMS) {
            c_sporo[i] = a.sporo; c_avail[i] = a.avail; c_cycle[i] = a.cycle; c_hbc[i] = a.hbc; c_batches[i] = a.batches;
          }
        }
      }
    }
    if (KEEP) c_flags[i] = fb;
    pk0 = __reduce_add_sync(0xffffffffu, pk0);
    pk1 = __reduce_add_sync(0xffffffffu, pk1);
    if (lane == 0) s_ent[k * kWarps + warp] = make_uint2(pk0, pk1);
  }
  if (EGGS) sa.acc.newEggs += t.newEggs;
  if (STATS) {
    sa.acc.bites += t.bites; sa.acc.infectBites += t.infectBites;
    sa.acc.cycles += t.cycles; sa.acc.sumCycles += t.sumCycles;
  }
  sa.acc.bad |= t.bad;
}

// Warp 0, after the tile's chunk counts are in s_ent: the tile's prefix table
// (the same 16-bit packed entries as the count pass's) into s_tab, and the
// tile's survivors of next state `lane` to lanes 0..7.
template <int I>
__device__ __forceinline__ uint32_t small_build_table(const uint2* s_ent, uint32_t* s_tab) {
  SAMPO_TILE_CONSTANTS(I);
  const int lane = threadIdx.x & 31;
  const uint2 e = lane < (int)kChunks ? s_ent[lane] : make_uint2(0u, 0u);
  uint32_t w[5], x[5];
  w[0] = (e.x & 0xffu) | ((e.x & 0xff00u) << 8);
  w[1] = ((e.x >> 16) & 0xffu) | ((e.x >> 8) & 0xff0000u);
  w[2] = (e.y & 0xffu) | ((e.y & 0xff00u) << 8);
  w[3] = ((e.y >> 16) & 0xffu) | ((e.y >> 8) & 0xff0000u);
  w[4] = ((e.x * 0x01010101u) >> 24) + ((e.y * 0x01010101u) >> 24);  // byte sums <= 32 cannot carry
#pragma unroll
  for (int q = 0; q < 5; q++) x[q] = w[q];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int q = 0; q < 5; q++) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x[q], o);
      if (lane >= o) x[q] += y;
    }
  }
  if (lane < (int)kChunks) {
#pragma unroll
    for (int q = 0; q < 5; q++) s_tab[lane * kPreEntryWords + q] = x[q] - w[q];
  }
  if (lane == (int)kChunks - 1) {
#pragma unroll
    for (int q = 0; q < 5; q++) s_tab[kChunks * kPreEntryWords + q] = x[q];
  }
  uint32_t tw = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t tq = __shfl_sync(0xffffffffu, x[q], kChunks - 1);
    if ((lane >> 1) == q) tw = (tq >> (16 * (lane & 1))) & 0xffffu;
  }
  return tw;
}

// Phase 2: the survivors of the tile in stage memory st (after
// small_update_tile<true, ...> and its table) to their slots in the next
// buffer: the tile's first slot of the state (s_d0) + the survivors of that
// state in earlier chunks (s_tab) + the rank within the chunk. A survivor
// whose slot falls outside its chunk's run sets tilebad and is not stored.
template <int I>
__device__ __forceinline__ void small_scatter_tile(bool whole, const uint8_t* st, const uint32_t* s_tab, const uint32_t* s_d0,
                                                   const DevPool& dst, uint32_t& tilebad) {
  SAMPO_TILE_CONSTANTS(I);
  const int tid = threadIdx.x, warp = tid >> 5;
  const float* c_age = (const float*)(st + 0 * kColBytes);
  const float* c_his = (const float*)(st + 1 * kColBytes);
  const float* c_delay = (const float*)(st + 2 * kColBytes);
  const float* c_sporo = (const float*)(st + 3 * kColBytes);
  const uint32_t* c_uni = (const uint32_t*)(st + 4 * kColBytes);
  const uint32_t* c_avail = (const uint32_t*)(st + 5 * kColBytes);
  const uint32_t* c_cycle = (const uint32_t*)(st + 6 * kColBytes);
  const uint32_t* c_hbc = (const uint32_t*)(st + 7 * kColBytes);
  const uint32_t* c_batches = (const uint32_t*)(st + 8 * kColBytes);
  const uint8_t* c_flags = st + 9 * kColBytes;
#pragma unroll
  for (int k = 0; k < kItems; k++) {
    const uint32_t i = k * kBlock + tid;
    const uint8_t fb = c_flags[i];
    const int b = fb == kGone ? 8 : (fb & 7);
    const uint32_t peers = __match_any_sync(0xffffffffu, (uint32_t)b);
    const uint32_t rk = __popc(peers & lanemask_lt());
    if (b < 8) {
      const uint32_t* e0 = s_tab + (k * kWarps + warp) * kPreEntryWords;
      const uint32_t* e1 = e0 + kPreEntryWords;
      const uint32_t sh = 16 * (b & 1);
      const uint32_t j = ((e0[b >> 1] >> sh) & 0xffffu) + rk;
      if (j < ((e1[b >> 1] >> sh) & 0xffffu)) {
        const uint32_t d = s_d0[b] + j;
        dst.age[d] = c_age[i]; dst.delay[d] = c_delay[i];
        dst.flags[d] = fb;
        if (!whole || b != EGG) dst.uni[d] = c_uni[i];
        if (!whole || b >= PUPA) dst.his[d] = c_his[i];
        if (!whole || b >= BMS) {
          dst.sporo[d] = c_sporo[i]; dst.avail[d] = c_avail[i]; dst.cycle[d] = c_cycle[i]; dst.hbc[d] = c_hbc[i];
          dst.batches[d] = c_batches[i];
        }
      } else {
        tilebad = 1;
      }
    }
  }
}

// What the CTAs tell each other of an hour (RepParams::smallRows): per tile its
// survivors by next state (16 bits each, 16 bytes), and per group of 16 tiles
// a record of 16 words that the CTAs of its tiles add to:
//   0-3  survivors by next state, 16 bits each   4  eggs laid
//   5 on  statistics of the next pool (SA_*; the youngest larva as the largest
//         SA_YOUNG - days, so that zero is the identity of every word)
// A CTA reads the groups' records and the tiles of its own group. (Every CTA
// reading 18 words of every tile took 2.3 us of an hour with three tiles,
// where its 27 reductions on every warp bound it, and 4 us with 300, where
// the L2 slices that hold the rows did; the hour went from 7.7 to 6.7 us and
// from 13.3 to 11.8 us.) Three sets of records rotate through the hours: the
// one in use, and the next, cleared meanwhile.
struct SmallRows {
  uint4* tiles;
  uint32_t* groups;    // [3][stride][16]
  uint32_t* state;     // the set the next launch starts with (all zero); records of the next one and of the one after that
                       // that may not be; whether a launch gave up waiting. Its records are not defined then, and the launches
                       // queued behind it do nothing, until the host has cleared them
  uint32_t stride;     // records of a set
};
constexpr uint32_t kGroupTiles = kSmallGroupTiles, kGroupWords = kSmallGroupWords, SA_YOUNG = 128;
__device__ __forceinline__ SmallRows small_rows(const RepParams& rp) {
  SmallRows r;
  r.stride = units_of(rp.smallTiles, kGroupTiles);
  r.groups = rp.smallRows;
  r.tiles = reinterpret_cast<uint4*>(r.groups + 3 * (size_t)r.stride * kGroupWords);
  r.state = reinterpret_cast<uint32_t*>(r.tiles + rp.smallTiles);
  return r;
}
// Phase 2, all threads: the survivors of tiles [0, t) into s_ex (two parts:
// the groups before t's, and the tiles before t in its own) and, with
// `totals`, those of all nold tiles, their eggs and the statistics into
// s_tot. Warp 0 reads the groups' records once, four lanes each (all CTAs read
// the same few lines, and the L2 slices that hold them serve them one after
// the other), warp 1 the tiles of t's group. Ends synchronised.
__device__ __forceinline__ void small_sum_rows(const SmallRows& rows, uint32_t set, uint32_t nold, uint32_t t, bool totals,
                                               uint32_t (*s_ex)[8], uint32_t* s_tot) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, gt = t / kGroupTiles, q = lane & 3u;
  auto unpack = [](const uint4& c, uint32_t (&v)[8]) {
    v[0] = c.x & 0xffffu; v[1] = c.x >> 16; v[2] = c.y & 0xffffu; v[3] = c.y >> 16;
    v[4] = c.z & 0xffffu; v[5] = c.z >> 16; v[6] = c.w & 0xffffu; v[7] = c.w >> 16;
  };
  if (warp == 0) {
    const uint4* g = reinterpret_cast<const uint4*>(rows.groups + (size_t)set * rows.stride * kGroupWords);
    const uint32_t lim = totals ? units_of(nold, kGroupTiles) : gt;
    uint32_t sum[8] = {0, 0, 0, 0, 0, 0, 0, 0}, ex[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // q = 0: survivors; else the record's words 4q on
    const bool widest = q == 3u;  // the youngest and oldest larva
#pragma unroll 1
    for (uint32_t j = lane >> 2; j < lim; j += 8u) {
      const uint4 c = __ldcg(g + (size_t)j * (kGroupWords / 4) + q);
      uint32_t v[8] = {c.x, c.y, c.z, c.w, 0u, 0u, 0u, 0u};
      if (q == 0u) unpack(c, v);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        sum[k] = widest ? max(sum[k], v[k]) : sum[k] + v[k];
        ex[k] += j < gt ? v[k] : 0u;
      }
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint32_t x = __shfl_xor_sync(0xffffffffu, sum[k], o);
        sum[k] = widest ? max(sum[k], x) : sum[k] + x;
        ex[k] += __shfl_xor_sync(0xffffffffu, ex[k], o);
      }
    }
    if (lane == 0u) {
#pragma unroll
      for (int k = 0; k < 8; k++) s_ex[0][k] = ex[k];
    }
    if (totals && lane < 4u) {
      if (widest) sum[0] = sum[0] ? SA_YOUNG - sum[0] : 0xffffffffu;
      // eggs laid and the statistics follow the survivors, as in the record
      uint32_t* to = s_tot + (q ? 4u + 4u * q : 0u);
#pragma unroll
      for (uint32_t k = 0; k < 8; k++)
        if (q == 0u || k < (widest ? 2u : 4u)) to[k] = sum[k];
    }
  } else if (warp == 1) {
    uint32_t v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (lane < t - gt * kGroupTiles) unpack(__ldcg(rows.tiles + gt * kGroupTiles + lane), v);
#pragma unroll
    for (int o = 1; o < (int)kGroupTiles; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0u) {
#pragma unroll
      for (int k = 0; k < 8; k++) s_ex[1][k] = v[k];
    }
  }
  __syncthreads();
}

// Phase 1's end: the CTA's statistics of the next pool (its tiles) to its
// row, in two halves around a CTA barrier: each warp's totals into s_red
// (every thread), then the CTA's totals out by the threads of warp `w` (the
// other warps may do other work meanwhile). ONE: the CTA has one tile, so that
// a warp's counts fit in 8 bits each (32 * I agents).
template <bool ONE>
__device__ __forceinline__ void small_stats_warps(const SmallAcc& sa, uint32_t (*s_red)[kSmallStats]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t v[kSmallStats] = {sa.l1, sa.fem, sa.inf, sa.acc.cycles, sa.acc.sumCycles, sa.acc.bites, sa.acc.infectBites,
                             sa.dmin, sa.dmax};
  if (ONE) {
    const uint32_t x = __reduce_add_sync(0xffffffffu, v[SA_FEM] | (v[SA_INF] << 8) | (v[SA_CYC] << 16) | (v[SA_BITES] << 24));
    v[SA_FEM] = x & 0xffu; v[SA_INF] = (x >> 8) & 0xffu; v[SA_CYC] = (x >> 16) & 0xffu; v[SA_BITES] = x >> 24;
  }
#pragma unroll
  for (int j = 0; j < (int)SA_DMIN; j++)
    if (!ONE || j == (int)SA_L1 || j == (int)SA_SUMCYC || j == (int)SA_IBITES) v[j] = __reduce_add_sync(0xffffffffu, v[j]);
  v[SA_DMIN] = __reduce_min_sync(0xffffffffu, v[SA_DMIN]);
  v[SA_DMAX] = __reduce_max_sync(0xffffffffu, v[SA_DMAX]);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < (int)kSmallStats; j++) s_red[warp][j] = v[j];
  }
}
__device__ __forceinline__ void small_stats_store(const SmallRows& rows, uint32_t set, uint32_t b, const uint32_t (*s_red)[kSmallStats], int w) {
  const uint32_t k = threadIdx.x - 32u * (uint32_t)w;
  if (k < kSmallStats) {
    uint32_t x = s_red[0][k];
#pragma unroll
    for (int i = 1; i < kWarps; i++) {
      const uint32_t y = s_red[i][k];
      x = k == SA_DMIN ? min(x, y) : k == SA_DMAX ? max(x, y) : x + y;
    }
    uint32_t* to = rows.groups + ((size_t)set * rows.stride + b / kGroupTiles) * kGroupWords + 5 + k;
    if (k == SA_DMIN) x = x == 0xffffffffu ? 0u : SA_YOUNG - x;
    if (x) {
      if (k >= SA_DMIN) atomicMax(to, x);
      else atomicAdd(to, x);
    }
  }
}
// Warp 0: tile t's survivors (tw: of next state `lane`, on lanes 0..7) and eggs.
__device__ __forceinline__ void small_counts_store(const SmallRows& rows, uint32_t set, uint32_t t, uint32_t tw, uint32_t eggs) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lo = __shfl_sync(0xffffffffu, tw, (2u * lane) & 7u), hi = __shfl_sync(0xffffffffu, tw, (2u * lane + 1u) & 7u);
  const uint32_t x = lane < 4u ? lo | (hi << 16) : eggs;
  if (lane < 4u) __stcg(reinterpret_cast<uint32_t*>(rows.tiles + t) + lane, x);
  if (lane < 5u && x) atomicAdd(rows.groups + ((size_t)set * rows.stride + t / kGroupTiles) * kGroupWords + lane, x);
}

// Every thread waits (bounded) for the bulk copies of the stage's tile;
// false for all when any wait ran out.
__device__ __forceinline__ bool small_wait_stage(uint64_t* bar, uint32_t& phase) {
  const bool ok = mbar_wait(bar, phase);
  phase ^= 1u;
  return __syncthreads_and(ok) != 0;
}

// One thread: the copies of slots [lo, lo + n) of the pool to the stage, the
// columns that hold a record of a state in them (whole: a narrow pool's).
template <int I>
__device__ __forceinline__ void small_issue_tile(const DevPool& src, const sampo_population& pop, bool whole, uint8_t* st, uint64_t* bar,
                                                 uint32_t lo, uint32_t n) {
  SAMPO_TILE_CONSTANTS(I);
  const uint32_t b4 = (n * 4 + 15) & ~15u, b1 = (n + 15) & ~15u;
  const bool uni = !whole || lo + n > pop.r[LARVA].start, his = !whole || lo + n > pop.r[PUPA].start,
             rest = !whole || lo + n > pop.r[BMS].start;
  mbar_arrive_tx(bar, (2u + (uni ? 1u : 0u) + (his ? 1u : 0u) + (rest ? 5u : 0u)) * b4 + b1);
  bulk_load(st + 0 * kColBytes, src.age + lo, b4, bar);
  bulk_load(st + 2 * kColBytes, src.delay + lo, b4, bar);
  bulk_load(st + 9 * kColBytes, src.flags + lo, b1, bar);
  if (uni) bulk_load(st + 4 * kColBytes, src.uni + lo, b4, bar);
  if (his) bulk_load(st + 1 * kColBytes, src.his + lo, b4, bar);
  if (rest) {
    bulk_load(st + 3 * kColBytes, src.sporo + lo, b4, bar);
    bulk_load(st + 5 * kColBytes, src.avail + lo, b4, bar);
    bulk_load(st + 6 * kColBytes, src.cycle + lo, b4, bar);
    bulk_load(st + 7 * kColBytes, src.hbc + lo, b4, bar);
    bulk_load(st + 8 * kColBytes, src.batches + lo, b4, bar);
  }
}

__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// The one-launch steps of p.reps[0] (a single simulation without a device
// seed stream): `nsteps` hourly steps in one cooperative launch (a day graph
// launches it once with 24). Per hour: the update (phase 1), whose per-tile
// counts and per-CTA statistics of the next pool go to rows in global
// memory; a grid barrier; the scatter (phase 2) and the arrival at a second
// grid barrier, after which every CTA computes the next hour's layout,
// statistics row, step constants and larval table itself from the same
// totals (the k_publish arithmetic; the last CTA, the one least likely to
// hold a tile, also writes them to the replicate's state for the host) before
// it waits there; then the next hour's tile copies go out. The constants
// of the launch's hours are prepared in shared memory at its start, one hour
// per thread (the host writes their inputs before the launch); only the
// biomass and the larval table wait for the hour's pool. The rows (SmallRows)
// are read through L2. The pool the scatter wrote with ordinary stores is
// read by the next hour's bulk copies after proxy fences.
template <int I>
__global__ void __launch_bounds__(kSmallThreads, kSmallMinBlocks) k_step_small(KParams p, uint32_t nsteps) {
  SAMPO_TILE_CONSTANTS(I);
  extern __shared__ __align__(128) uint8_t stage[];
  __shared__ StepCtx s_c;
  __shared__ ModelConst s_mc;
  __shared__ uint32_t s_kill[100];
  __shared__ sampo_population s_pop;
  __shared__ StepCtx s_ctx[kSmallHours];
  __shared__ __align__(8) uint64_t s_mbar;
  __shared__ uint2 s_ent[kChunks];
  __shared__ __align__(16) uint32_t s_tab[(kChunks + 1) * kPreEntryWords];
  __shared__ uint32_t s_ex[2][8], s_tot[kSmallRows + kSmallStats], s_d0[8], s_ne[kWarps];
  __shared__ uint32_t s_red[kWarps][kSmallStats];
  __shared__ uint32_t s_flag, s_ok, s_last;
  __shared__ uint32_t s_active, s_end, s_nold, s_cur, s_cap, s_step, s_stop;
  __shared__ float s_cc;
  const RepParams& rp = p.reps[0];
  SimDev* sim = rp.sim;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t G = gridDim.x, b = blockIdx.x;
  uint32_t phase = 0, barriers = 0;
  bool met = true, ok = true;
  __shared__ SmallRows rows;            // (in shared memory: registers are short)
  __shared__ uint32_t s_set, s_dirty[3];  // the set in use; records of the next one (1) and the one after (2) that may not be zero
  const bool whole = !p.wide;     // ages are whole hours (state_cols)

  // ---- the replicate's state at the launch (the previous kernel wrote it) ----
  if (tid == 0) {
    mbar_init(&s_mbar);
    fence_mbar_init();
    rows = small_rows(rp);
    const uint32_t gave_up = __ldcg(rows.state + 3), active = gave_up ? 0u : sim->active;
    if (gave_up && b == 0) atomicOr(&sim->error, SAMPO_DEV_ERR_BARRIER);
    s_set = __ldcg(rows.state);
    s_dirty[1] = __ldcg(rows.state + 1);
    s_dirty[2] = __ldcg(rows.state + 2);
    s_pop = sim->pop;
    s_active = active;
    s_end = active ? s_pop.r[GRAVID].end : 0u;
    s_nold = (s_end + kTile - 1) / kTile;
    s_cur = sim->cur;
    s_cap = sim->capacity;
    s_step = sim->step;
    s_stop = sim->stop_step;
    s_cc = sim->cc;
    if (b < s_nold) {
      const uint32_t lo = b * kTile;
      small_issue_tile<I>(rp.pool[s_cur], s_pop, whole, stage, &s_mbar, lo, min((uint32_t)kTile, s_end - lo));
    }
  }
  copy16(&s_c, &sim->ctx[sim->step & 1u], (int)sizeof(StepCtx), tid, blockDim.x);
  for (int k = tid; k < 100; k += blockDim.x) s_kill[k] = sim->larvaKill[sim->step & 1u][k];
  load_model_const(p.mc, s_mc);
  __syncthreads();
  if (tid == 0) s_c.larvaKill = s_kill;
  // the constants of the steps that follow the launch's hours, but for their pool's biomass
  nsteps = min(nsteps, kSmallHours);
  for (uint32_t j = tid; j < nsteps; j += blockDim.x) {
    CtxInputs in;
    load_ctx_inputs(rp, s_step + 1u + j, in);
    StepCtx c;
    make_ctx(in, s_kill, s_pop, c);
    s_ctx[j] = c;
  }
  __syncthreads();

  for (uint32_t hour = 0; hour < nsteps; hour++) {
    if (!s_active) break;  // stopped or paused (uniform)
    const uint32_t nold = s_nold, end = s_end;
    SmallAcc sa;
    sa.acc = Acc{0, 0, 0, 0, 0, 0};
    sa.l1 = sa.fem = sa.inf = sa.dmax = sa.devoob = sa.tilebad = 0;
    sa.dmin = 0xffffffffu;

    const uint32_t set = s_set, stale = s_dirty[1];

    // ---- phase 1: decide (and, for tile b, finish) every tile of this CTA ----
    if (nold > G && b < nold) {
      // more tiles than CTAs: count tile b (its copies are on their way)
      // without keeping it, then the other tiles of this CTA one after the
      // other in the stage, then load tile b again and keep it
      ok = small_wait_stage(&s_mbar, phase);
      for (uint32_t t = b; t < nold && ok; t += G) {
        if (t != b) {
          if (tid == 0) {
            fence_proxy_async();
            small_issue_tile<I>(rp.pool[s_cur], s_pop, whole, stage, &s_mbar, t * kTile, min((uint32_t)kTile, end - t * kTile));
          }
          ok = small_wait_stage(&s_mbar, phase);
          if (!ok) break;
        }
        const uint32_t eggs_before = sa.acc.newEggs;
        small_update_tile<I, false, true, true>(s_c, s_mc, s_pop, whole, stage, t * kTile, end, s_ent, sa);
        const uint32_t ne = __reduce_add_sync(0xffffffffu, sa.acc.newEggs - eggs_before);
        if (lane == 0) s_ne[warp] = ne;
        __syncthreads();
        if (warp == 0) {
          const uint32_t tw = small_build_table<I>(s_ent, s_tab);
          uint32_t e = lane < kWarps ? s_ne[lane] : 0u;
          e = __reduce_add_sync(0xffffffffu, e);
          small_counts_store(rows, set, t, tw, e);
        }
        __syncthreads();  // the stage is read before the next copy overwrites it
      }
      if (ok) {
        if (tid == 0) {
          fence_proxy_async();
          small_issue_tile<I>(rp.pool[s_cur], s_pop, whole, stage, &s_mbar, b * kTile, min((uint32_t)kTile, end - b * kTile));
        }
        ok = small_wait_stage(&s_mbar, phase);
        if (ok) {
          small_update_tile<I, true, false, false>(s_c, s_mc, s_pop, whole, stage, b * kTile, end, s_ent, sa);  // counted above
          small_stats_warps<false>(sa, s_red);
          __syncthreads();
          if (warp == 0) (void)small_build_table<I>(s_ent, s_tab);
          else if (warp == 1) small_stats_store(rows, set, b, s_red, 1);
        }
      }
    } else if (b < nold) {
      ok = small_wait_stage(&s_mbar, phase);
      if (ok) {
        const uint32_t eggs_before = sa.acc.newEggs;
        small_update_tile<I, true, true, true>(s_c, s_mc, s_pop, whole, stage, b * kTile, end, s_ent, sa);
        const uint32_t ne = __reduce_add_sync(0xffffffffu, sa.acc.newEggs - eggs_before);
        if (lane == 0) s_ne[warp] = ne;
        small_stats_warps<true>(sa, s_red);
        __syncthreads();
        if (warp == 0) {  // the tile's table and counts
          const uint32_t tw = small_build_table<I>(s_ent, s_tab);
          uint32_t e = lane < kWarps ? s_ne[lane] : 0u;
          e = __reduce_add_sync(0xffffffffu, e);
          small_counts_store(rows, set, b, tw, e);
        } else if (warp == 1) {  // meanwhile the CTA's statistics
          small_stats_store(rows, set, b, s_red, 1);
        }
      }
    }
    if (tid == 0) s_ok = ok ? 1u : 0u;

    // ---- grid barrier A: every tile's counts and every CTA's statistics are published ----
    met = small_grid_barrier(&p.bat->bar, G * ++barriers, &s_flag);
    ok = s_ok != 0;  // this CTA's copies all landed

    // ---- phase 2: totals, next layout, this tile's first slots; scatter ----
    small_sum_rows(rows, set, nold, b < nold ? b : nold, true, s_ex, s_tot);
    {  // the next hour's records (nobody has read them since the hour before the last)
      const uint32_t n = set == 2u ? 0u : set + 1u;
      uint32_t* next = rows.groups + (size_t)n * rows.stride * kGroupWords;
      for (uint32_t i = b * blockDim.x + tid; i < stale * kGroupWords; i += G * blockDim.x) __stcg(next + i, 0u);
      if (tid == 0) {  // (read again past the next CTA barrier at the earliest)
        s_set = n;
        s_dirty[1] = s_dirty[2];
        s_dirty[2] = units_of(nold, kGroupTiles);
      }
    }
    uint32_t tot[8], base[8];
#pragma unroll
    for (int k = 0; k < 8; k++) tot[k] = s_tot[k];
    const uint32_t ne = s_tot[8];
    const bool fits = layout_fits(tot, ne, s_cap);
    sampo_population np;
    next_layout(tot, ne, np, base);
    const bool write = ok && met && fits;
    const DevPool dst = rp.pool[s_cur ^ 1u];
    if (write && b < nold) {
      // (by constant indexes: base stays in registers)
      uint32_t mine = base[0];
#pragma unroll
      for (int k = 1; k < 8; k++) mine = tid == k ? base[k] : mine;
      if (tid < 8) s_d0[tid] = mine + s_ex[0][tid] + s_ex[1][tid];
      __syncthreads();
      small_scatter_tile<I>(whole, stage, s_tab, s_d0, dst, sa.tilebad);
      // more tiles than CTAs: the other tiles of this CTA, loaded and updated again
      for (uint32_t t = b + G; t < nold; t += G) {
        __syncthreads();  // the stage is read
        if (tid == 0) {
          fence_proxy_async();
          small_issue_tile<I>(rp.pool[s_cur], s_pop, whole, stage, &s_mbar, t * kTile, min((uint32_t)kTile, end - t * kTile));
        }
        if (!small_wait_stage(&s_mbar, phase)) { ok = false; break; }
        small_update_tile<I, true, false, false>(s_c, s_mc, s_pop, whole, stage, t * kTile, end, s_ent, sa);
        small_sum_rows(rows, set, nold, t, false, s_ex, s_tot);
        if (warp == 0) {
          const uint32_t tw = small_build_table<I>(s_ent, s_tab);
          // the update again must give the counts of phase 1
          if (lane < 8 && tw != ((__ldcg(reinterpret_cast<const uint32_t*>(rows.tiles + t) + lane / 2) >> (16 * (lane & 1))) & 0xffffu))
            sa.tilebad = 1;
          uint32_t mine = base[0];
#pragma unroll
          for (int k = 1; k < 8; k++) mine = lane == k ? base[k] : mine;
          if (lane < 8) s_d0[lane] = mine + s_ex[0][lane] + s_ex[1][lane];
        }
        if (__syncthreads_or(sa.tilebad)) break;
        small_scatter_tile<I>(whole, stage, s_tab, s_d0, dst, sa.tilebad);
      }
    }
    if (write) {
      // new eggs at [0, newEggs) of the next buffer, egg tile e on CTA G-1-(e mod G)
      const uint32_t negg = (ne + kTile - 1) / kTile;
      for (uint32_t e = G - 1 - b; e < negg; e += G) {
#pragma unroll
        for (int k = 0; k < kItems; k++) {
          const uint32_t id = e * kTile + k * kBlock + tid;
          if (id < ne) {
            Rec a;
            new_egg(s_c, id, a);
            dst.age[id] = a.age; dst.delay[id] = a.delay;
            if (!whole) {
              dst.his[id] = a.his; dst.sporo[id] = a.sporo; dst.uni[id] = a.uni; dst.avail[id] = a.avail;
              dst.cycle[id] = a.cycle; dst.hbc[id] = a.hbc; dst.batches[id] = a.batches;
            }
            dst.flags[id] = (uint8_t)(EGG | (a.female << 3));
          }
        }
      }
    }
    fence_proxy_async_global();  // the next hour reads these stores with bulk copies

    // ---- this CTA's error bits (the capacity bit from CTA 0 only) ----
    {
      uint32_t x = (sa.acc.bad ? SAMPO_DEV_ERR_LARVATABLE : 0u) | (sa.tilebad ? SAMPO_DEV_ERR_TILECOUNT : 0u) |
                   (sa.devoob ? SAMPO_DEV_ERR_DEVRATES : 0u) | (ok ? 0u : SAMPO_DEV_ERR_TMA) |
                   (met ? 0u : SAMPO_DEV_ERR_BARRIER) | (fits ? 0u : SAMPO_DEV_ERR_CAPACITY);
      x = __reduce_or_sync(0xffffffffu, x);
      if (b != 0) x &= ~SAMPO_DEV_ERR_CAPACITY;
      if (lane == 0 && x) atomicOr(&sim->error, x);
    }
    if (!met || !ok) break;  // the error bits are set; nothing after this hour is valid
    if (!fits) {
      // the next layout does not fit: the replicate pauses at this step with
      // its pool and constants (k_publish does the same for the three-kernel step)
      if (b == G - 1u && tid == 0) sim->active = 0;
      break;
    }

    // ---- the next hour's state (the k_publish arithmetic, publish_rep), by
    //      every CTA from the same totals, between its arrival at the grid
    //      barrier (its stores are in) and its wait there ----
    const uint32_t step = s_step + 1u;
    const bool active = step < s_stop;
    const bool more = hour + 1u < nsteps && active;  // another hour in this launch
    if (more) small_grid_arrive(&p.bat->bar);
    const uint32_t next_end = np.r[GRAVID].end, next_nold = (next_end + kTile - 1) / kTile;
    const uint32_t* st = s_tot + kSmallRows;
    // the next pool's statistics (kernel/calcL1de.cl:259-280, calcGender.cl)
    np.numLarvae1DayEquiv = (np.r[LARVA].end > np.r[LARVA].start) ? st[SA_L1] : 0u;
    np.numFemale = st[SA_FEM];
    np.numPotentiallyInfective = st[SA_INF];
    __syncthreads();  // every thread is past its last read of s_c, s_kill and s_pop
    if (tid == 0) {
      const uint32_t biomass = np.numLarvae1DayEquiv + np.r[EGG].end + (np.r[PUPA].end - np.r[PUPA].start);
      s_c.totalBiomass = biomass;
      if (b == G - 1u) {
        // the replicate's state and the coming step's row for the host
        sampo_bites_cycles nbnc;
        nbnc.numCyclesReported = st[SA_CYC];
        nbnc.sumCyclesReported = st[SA_SUMCYC];
        nbnc.numBitesReported = st[SA_BITES];
        nbnc.numInfectBitesReported = st[SA_IBITES];
        // the reference's shared empty initial ranges (src/abms.c:204-219)
        bool shared_end = false;
        uint32_t moved = 0;
        for (int k = 1; k < 8; k++) {
          shared_end |= s_pop.r[k].end == s_pop.r[k - 1].end;
          moved += s_tot[k];
        }
        if (shared_end && moved) sim->warn = __ldcg(&sim->warn) | SAMPO_DEV_WARN_REF_LAYOUT;
        sim->ctx[step & 1u].totalBiomass = biomass;
        sim->ctx[step & 1u].larvaKill = sim->larvaKill[step & 1u];
        sim->pop = np;
        sim->bnc = nbnc;
        sim->step = step;
        sim->cur = s_cur ^ 1u;
        sampo_stats_row row;
        row.pop = np;
        row.bnc = nbnc;
        rp.rows[step % rp.ring] = row;
        if (!active) sim->active = 0;
      }
      s_pop = np;
      s_step = step;
      s_cur ^= 1u;
      s_end = next_end;
      s_nold = next_nold;
      s_active = active;
    }
    if (warp == kWarps - 1) {  // the next hour's constants (the last CTA also stores them)
      const StepCtx& c = s_ctx[hour];
      const uint32_t* from = reinterpret_cast<const uint32_t*>(&c);
      const uint32_t bio = (uint32_t)(&c.totalBiomass - from), tab = (uint32_t)(reinterpret_cast<const uint32_t*>(&c.larvaKill) - from);
      uint32_t* const to = reinterpret_cast<uint32_t*>(&s_c);
      uint32_t* const out = reinterpret_cast<uint32_t*>(&sim->ctx[step & 1u]);
      for (uint32_t k = lane; k < sizeof(StepCtx) / 4; k += 32u) {
        if (k == bio) continue;
        to[k] = from[k];
        if (b == G - 1u && k != tab && k != tab + 1u) out[k] = from[k];
      }
    } else {  // the next hour's larval table (every CTA; the last one also stores it)
      const uint32_t dmin = st[SA_DMIN], dmax = st[SA_DMAX], l1 = np.numLarvae1DayEquiv;
      for (int d = tid - 32; d >= 0 && d < 100; d += blockDim.x - 64) {
        const uint32_t k = larva_kill_entry((uint32_t)d, dmin, dmax, l1, s_cc);
        s_kill[d] = k;
        if (b == G - 1u) sim->larvaKill[step & 1u][d] = k;
      }
    }
    if (!more) break;  // (no copy is in flight)

    // ---- the grid barrier's wait: every CTA's stores are in; the next hour's tile ----
    met = small_grid_wait(&p.bat->bar, G * ++barriers, &s_flag);
    if (!met) break;
    if (tid == 0 && b < next_nold) {
      fence_proxy_async_global();
      fence_proxy_async();
      small_issue_tile<I>(dst, s_pop, whole, stage, &s_mbar, b * kTile, min((uint32_t)kTile, next_end - b * kTile));
    }
  }
  if (!met && tid == 0) atomicOr(&sim->error, SAMPO_DEV_ERR_BARRIER);
  if ((!met || !ok) && tid == 0) __stcg(rows.state + 3, 1u);
  // a copy that did not land in time may still be in flight: let it land
  // (bounded) before the CTA can exit
  if (tid == 0 && !ok) (void)mbar_wait(&s_mbar, phase ^ 1u);  // the phase whose wait ran out

  // ---- the last CTA out rearms the barrier for the next launch ----
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_last = atomicAdd(&p.bat->done, 1u) == G - 1u ? 1u : 0u;
    if (s_last) {
      p.bat->bar = 0u;
      p.bat->done = 0u;
      rows.state[0] = s_set;
      rows.state[1] = s_dirty[1];
      rows.state[2] = s_dirty[2];
    }
  }
}

}  // namespace sampo
