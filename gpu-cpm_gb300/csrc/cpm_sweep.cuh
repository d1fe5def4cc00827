// cpm_sweep.cuh — the checkerboard Metropolis sweep, instantiated for 2D
// (cpm_sweep2d.cu) and 3D (cpm_sweep3d.cu).
//
//   sweep_kernel<NDIM, KR, MODE, BATCH>  persistent over all MCS of a run.
//                              Replaces copyAttempt (src/kernels2d.cu:44-583)
//                              and copyAttempt3d (src/kernels3d.cu:51-594).
//
// Schedule.  Sites are coloured by their class on every axis (even / odd /
// last coordinate of an odd axis); one phase ("slot") is one colour, and one
// MCS runs every non-empty slot in lexicographic (cz, cy, cx) order.  All
// targets of a slot are >= 2 apart on each axis, so an attempt never reads a
// site another attempt of the same slot may write; the cell tables are read
// as they stood when the slot began (double-buffered, see cpm_internal.h) and
// the integer deltas are exact and order-free.  The result is independent of
// thread, block and replica order, and the CPU oracle reproduces it bit for
// bit.
//
// A warp takes tasks of 32 target columns x `rows` target rows:
//   1. draw: KR rows at a time, every lane draws for its targets (KR Philox
//      chains side by side) and reads the target and the drawn source.  A
//      source of the target's own value ends the attempt; the others go on
//      the warp's queue with both values.
//   2. evaluate: whenever 32 attempts are queued, dH, Metropolis test,
//      lattice write and table deltas, one attempt per lane.  What a warp has
//      left when its tasks are done is pooled with the other warps' of the
//      block, so that even a phase of few targets evaluates full batches.
//
// Nothing is staged: sites are read through the L1 cache, which holds what
// the draws of a task's rows brought in when its attempts are evaluated.  A
// phase's reads are of sites no other attempt of the phase writes, and the
// acquire of the phase barrier (which drops the SM's L1 lines) orders them
// after the writes of the phases before, so plain loads see them.  Against
// warp tiles staged in shared memory (by cp.async.bulk.tensor, or a load and
// a store per site), which needed a boundary test of every target before its
// draw to keep the staging worth its while: 256^3 tissue, 20 MCS, 6.72 ->
// 3.61 ms; 4096^2 tissue, 50 MCS, 8.44 -> 7.65 ms; a 101 x 75 x 61 box, 20
// MCS, 5.09 -> 2.84 ms.
//
// Bound: instruction issue on large lattices (6 warp instructions per
// attempt in 2D, 10 in 3D), the chain of one warp through a phase on small ones: draw,
// two L2 round trips, ~400 instructions, the grid barrier (2,600 cycles, 3,200
// with reductions outstanding).
//
// Launches (SweepArgs::block_local): grid dispatch deals the tasks of a slot
// to all blocks, block b taking tasks b, b + G, b + 2G, ..., each row of tasks
// rotated by its row index; a block's warps claim them from a shared counter.
// One grid barrier ends each phase.  BATCH kernels do so over all replicas of
// a batch.  Replica dispatch lets each block claim whole replicas and run all
// their phases with block barriers.
#pragma once

#include <cstdint>

#include "cpm_device.cuh"
#include "cpm_sweep_common.cuh"

namespace gpucpm {
namespace {

// What a kernel carries besides the plain terms.
constexpr int kPlain = 0;
constexpr int kExt = 1;    // act, 3D persistence
constexpr int kScore = 2;  // likelihood-ratio scores (2D)
constexpr int kOne = 3;    // kExt with one lattice copy (SweepArgs::lat2 is null)

// Warps per block (one block per SM): 24 at 80 registers for the plain 2D
// sweep, 20 at 96 for the others, which would spill at 80.  (28 or 32 warps at
// 72 or 64 registers: 4096^2 tissue 7.96 -> 8.13 or 8.54 ms.)
template <int NDIM, int KR, int MODE, bool BATCH>
__host__ __device__ constexpr int sweep_warps() {
  return NDIM == 2 && MODE == kPlain && !BATCH ? 24 : 20;
}

// An attempt to evaluate: target site, random word (its upper 24 bits) with
// the source's direction (lower 8), source and target values.
struct alignas(16) Attempt {
  uint32_t site, draw, s, t;
};

template <int KR>
__host__ __device__ constexpr int queue_len() {
  return 32 + 32 * KR;
}

// A changed table row: row, target site, the row's area, perimeter change + 64
// and (bit 8) whether the cell lost the site.
struct alignas(16) RowChange {
  uint32_t row, site, area, change;
};
constexpr int kChangeLen = 32 + 64;

// Whether a kernel queues the row changes of accepted copies and makes them 32
// at a time.  Few lanes of a batch accept (one in eight on the tissues), and
// the ~250 instructions of a copy's row changes ran for every batch: 4096^2
// tissue, 50 MCS 7.65 -> 7.07 ms.  In the kernels of small lattices a phase is
// one warp's chain, which a second queue lengthens; it gained nothing in 3D
// (3.61 ms either way) and lost where many accept (256 ragged replicas 22.9 ->
// 23.7 ms, scores 31.6 -> 32.4).
template <int NDIM, int KR, int MODE, bool BATCH>
__host__ __device__ constexpr bool defers() {
  return NDIM == 2 && KR == 4 && MODE == kPlain && !BATCH;
}
template <int NDIM, int KR, int MODE, bool BATCH>
__host__ __device__ constexpr int warp_smem() {
  return (int)sizeof(Attempt) * (32 + queue_len<KR>()) +
         (defers<NDIM, KR, MODE, BATCH>() ? (int)sizeof(RowChange) * kChangeLen : 0);
}

// Dirty-list entries of a phase kept in shared memory (the rest in global
// memory): a 4096^2 tissue pushes ~1,000 per block and phase.
constexpr unsigned kListSmem = 2048;

// What attempts need of their replica, in shared memory (one for the block,
// in batches one per warp): kept in registers it made every kernel spill.
struct ReplicaCtx : DevReplica, ParamHead {
  const DevParams* P;
  int rep;
};

// Act model (src/kernels2d.cu:338-473, src/kernels3d.cu:347-470): the
// geometric mean of max(amax + act[i] - tick, 0) over site (x, y, z) and
// those of its neighbours that hold `id`, as exp2 of the mean log2 (own
// log2_pos / exp2_own, summed in neighbour order); 0 when a factor is 0.
// L and A are the replica's lattice and act stamps as they stood when the
// phase began.
template <int NDIM>
__device__ __forceinline__ float act_mean(const uint32_t* L, const uint32_t* A, int x, int y,
                                          int z, int nx, int ny, int nz, uint32_t id, int amax,
                                          long long tick) {
  auto at = [&](int xx, int yy, int zz) { return ((long long)zz * ny + yy) * nx + xx; };
  const long long a0 = (long long)amax + (long long)A[at(x, y, z)] - tick;
  if (a0 <= 0) return 0.0f;
  float sum = log2_pos((float)a0);
  int count = 1;
  const int zlo = NDIM == 3 ? -1 : 0, zhi = NDIM == 3 ? 1 : 0;
  for (int dz = zlo; dz <= zhi; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        if (!dz && !dy && !dx) continue;
        const long long n = at(wrap_coord(x + dx, nx), wrap_coord(y + dy, ny),
                               NDIM == 3 ? wrap_coord(z + dz, nz) : 0);
        if (L[n] != id) continue;
        const long long v = (long long)amax + (long long)A[n] - tick;
        if (v <= 0) return 0.0f;
        sum = __fadd_rn(sum, log2_pos((float)v));
        ++count;
      }
  return exp2_own(__fdiv_rn(sum, (float)count));
}

// Warp-reduces a lane's score partial sums and adds them, by lane 0, to the
// (replica, MCS) row of the score buffer: J pairs at their index, then
// lambda_area, lambda_perim and T in that order when enabled.  Clears the
// partial sums.
__device__ __forceinline__ void flush_scores(const SweepArgs& a, float* sc, int rep,
                                             unsigned long long tick) {
#pragma unroll
  for (int k = 0; k < kScoreRegs; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sc[k] += __shfl_xor_sync(kFull, sc[k], o);
  const long long row = (long long)tick - (long long)a.score_base;
  if ((threadIdx.x & 31) == 0 && rep >= 0 && row >= 0 && row < a.score_len) {
    float* dst = a.scores + ((long long)rep * a.score_len + row) * kScoreMax;
    int k = 0;
#pragma unroll
    for (int p = 0; p < kScorePairsMax; ++p)
      if (p < a.score_spec.n_pairs) atomicAdd(dst + k++, sc[p]);
    if (a.score_spec.lambda_area) atomicAdd(dst + k++, sc[kScorePairsMax]);
    if (a.score_spec.lambda_perim) atomicAdd(dst + k++, sc[kScorePairsMax + 1]);
    if (a.score_spec.temperature) atomicAdd(dst + k++, sc[kScorePairsMax + 2]);
  }
#pragma unroll
  for (int k = 0; k < kScoreRegs; ++k) sc[k] = 0.0f;
}

// Entry j of the block's list of the running phase's copies in act runs with
// one lattice (SweepArgs::pend).
__device__ __forceinline__ unsigned long long& pend_site(const SweepArgs& a, unsigned j) {
  return reinterpret_cast<unsigned long long*>(a.pend)[(long long)blockIdx.x * a.pend_cap + j];
}
__device__ __forceinline__ uint32_t& pend_value(const SweepArgs& a, unsigned j) {
  return reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned long long*>(a.pend) +
                                     (long long)gridDim.x * a.pend_cap)
      [(long long)blockIdx.x * a.pend_cap + j];
}

// LOCAL: for replica dispatch, where the kernel differs (see s_pt).
template <int NDIM, int KR, int MODE, bool BATCH, bool LOCAL>
__global__ void __launch_bounds__((32 * sweep_warps<NDIM, KR, MODE, BATCH>()), 1)
    sweep_kernel(const __grid_constant__ SweepArgs a) {
  constexpr bool ONE = MODE == kOne, EXT = MODE == kExt || ONE, SCORE = MODE == kScore;
  constexpr int NB = NDIM == 2 ? 8 : 26, NBC = NB + 1;
  constexpr int QLEN = queue_len<KR>();
  constexpr bool DEFER = defers<NDIM, KR, MODE, BATCH>();
  constexpr bool SHARED_PT = DEFER && !LOCAL;
  constexpr unsigned long long NSLOTS = NDIM == 2 ? 9 : 27;
  // the pooled attempts (32 per warp), then the warps' queues
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_list[2][kListSmem];
  __shared__ float s_J[BATCH ? 1 : kMaxTypes * kJPitch];
  __shared__ TypeParams s_type[BATCH ? 1 : kMaxTypes];
  __shared__ ReplicaCtx s_ctx[BATCH ? sweep_warps<NDIM, KR, MODE, BATCH>() : 1];
  __shared__ int s_ok, s_claim;
  __shared__ unsigned s_cnt[2], s_next[2], s_pool, s_pend[2];
  __shared__ unsigned long long s_tick0;
  // A phase's table pointers.  Where row changes are queued few instructions use
  // them, and the twelve registers do more for the rest (4096^2, 50 MCS 6.69 ->
  // 6.47 ms).  Elsewhere every accepted copy would wait for them (256 ragged
  // replicas 16.6 -> 18.9 ms, 1001 x 777 0.87 -> 0.93), and in replica dispatch a
  // block's few rows change often (512 x 256^2 of small cells, 50 MCS 34.0 -> 39.1).
  __shared__ PhaseTables<NDIM> s_pt[SHARED_PT ? 2 : 1];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wpb = blockDim.x >> 5;
  Attempt* const pool = reinterpret_cast<Attempt*>(smem_raw);
  Attempt* const queue = pool + wpb * 32 + warp * QLEN;
  RowChange* const changes = reinterpret_cast<RowChange*>(pool + wpb * (32 + QLEN)) +
                             warp * kChangeLen;  // (DEFER)
  int nchange = 0;  // queued row changes
  const uint32_t k0 = (uint32_t)a.seed, k1 = (uint32_t)(a.seed >> 32);
  int* err = reinterpret_cast<int*>(&a.ctl[kCtlErr]);
  // A phase's dirty list: the first kListSmem entries in shared memory, the
  // others at their index in the block's global list.
  auto blist = [&](int b) { return a.dlist + (2LL * blockIdx.x + b) * a.list_cap; };
  unsigned episode = 0;
  unsigned n_eval = 0, n_acc = 0;  // of replica r, warp-uniform
  float sc[kScoreRegs];  // (scores) the lane's sums of replica r at the running MCS
#pragma unroll
  for (int k = 0; k < kScoreRegs; ++k) sc[k] = 0.0f;
  if (tid < 2) s_cnt[tid] = s_next[tid] = s_pend[tid] = 0;
  if (tid == 0) s_pool = 0;
  auto tables_of = [&](const int cur) -> PhaseTables<NDIM> {
    return {cur ? a.ap[1] : a.ap[0], cur ? a.cs[1] : a.cs[0],   cur ? a.ap[0] : a.ap[1],
            cur ? a.cs[0] : a.cs[1], cur ? a.dap[1] : a.dap[0], cur ? a.dcs[1] : a.dcs[0]};
  };
  if (SHARED_PT && tid < 2) s_pt[tid] = tables_of(tid);
  // Every block reads *tick_ptr before its first barrier arrival, and block
  // 0 advances it only after its last barrier, so all blocks see one value.
  if (tid == 0) s_tick0 = a.tick_ptr ? __ldcg(a.tick_ptr) : a.tick0;
  __syncthreads();

  // ---- the replica at hand ------------------------------------------------
  ReplicaCtx& ctx = s_ctx[BATCH ? warp : 0];
  int r = -1;
  // by a whole warp, a word per lane: every task of a batch begins with it,
  // and one lane's loads of the fields took ~60 instructions and as many
  // trips as fields (with the search below and four rows side by side: 256
  // ragged replicas, 20 MCS 17.4 -> 16.4 ms; 128 of 128^2 to 512^2 5.72 -> 5.29)
  auto load_replica = [&](int rep) {
    constexpr int kRep = sizeof(DevReplica) / 4, kHead = sizeof(ParamHead) / 4;
    const uint32_t v =
        lane < kRep ? __ldg(reinterpret_cast<const uint32_t*>(a.reps + rep) + lane) : 0u;
    const DevParams* P = a.params + __shfl_sync(kFull, v, offsetof(DevReplica, pset) / 4);
    const uint32_t h =
        lane < kHead
            ? __ldg(reinterpret_cast<const uint32_t*>(static_cast<const ParamHead*>(P)) + lane)
            : 0u;
    if (lane < kRep) reinterpret_cast<uint32_t*>(static_cast<DevReplica*>(&ctx))[lane] = v;
    if (lane < kHead) reinterpret_cast<uint32_t*>(static_cast<ParamHead*>(&ctx))[lane] = h;
    if (lane == 0) ctx.P = P, ctx.rep = rep;
  };
  auto flush_counters = [&]() {
    if (lane == 0 && r >= 0) {
      if (n_eval) atomicAdd(&a.counters[2 * r], (unsigned long long)n_eval);
      if (n_acc) atomicAdd(&a.counters[2 * r + 1], (unsigned long long)n_acc);
    }
    n_eval = n_acc = 0;
  };

  // Deltas of the phase with double-buffer index `prv` into the copy it read
  // and, in act runs, its copies.  Where the tables have few rows for the
  // lattice's sites (a.scan) every row is looked at, one thread each, with
  // coalesced loads; elsewhere the rows of this block's dirty list, each
  // delta taken with an exchange, so that a row listed twice is replayed once.
  // The list costs a shared-memory atomic and stores per batch and three
  // exchanges per entry, and the busiest cells are on it many times (list /
  // scan: 256 ragged replicas, 20 MCS 23.1 / 17.4 ms; gradient of 128 x 256^2
  // 31.5 / 24.8 ms; act on 512^2 2.03 / 1.90 ms; 4096^2 tissue 7.08 / 7.06 ms).
  auto replay_phase = [&](int prv, unsigned first) {
    unsigned long long* const dap = prv ? a.dap[1] : a.dap[0];
    unsigned long long* const ap = prv ? a.ap[1] : a.ap[0];
    unsigned long long* const dcs =
        reinterpret_cast<unsigned long long*>(prv ? a.dcs[1] : a.dcs[0]);
    unsigned long long* const cs = reinterpret_cast<unsigned long long*>(prv ? a.cs[1] : a.cs[0]);
    if (a.scan) {
      // every row of the launch, each by one thread of the grid (of the block
      // in replica dispatch)
      const unsigned n = BATCH ? a.scan_rows : (unsigned)ctx.ncells + 1u;
      const unsigned row0 = BATCH ? 0u : (unsigned)ctx.cell_off;
      const bool local = !BATCH && a.block_local;
      const unsigned stride = local ? blockDim.x : blockDim.x * gridDim.x;
      for (unsigned j = first + (local ? 0u : blockIdx.x * blockDim.x); j < n; j += stride) {
        const long long row = row0 + j;
        unsigned long long d[NDIM + 1];
        d[NDIM] = __ldcg(dap + row);
        if constexpr (NDIM == 2) {
          const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(dcs) + row);
          d[0] = v.x, d[1] = v.y;
        } else {
#pragma unroll
          for (int k = 0; k < NDIM; ++k) d[k] = __ldcg(dcs + row * NDIM + k);
        }
        if (d[NDIM]) {
          __stcg(dap + row, 0ull);
          atomicAdd(ap + row, d[NDIM]);
        }
#pragma unroll
        for (int k = 0; k < NDIM; ++k)
          if (d[k]) {
            __stcg(dcs + row * NDIM + k, 0ull);
            atomicAdd(cs + row * NDIM + k, d[k]);
          }
      }
    } else {
      const unsigned n = min(s_cnt[prv], (unsigned)a.list_cap);  // see kErrListFull
      for (unsigned j = first; j < n; j += blockDim.x) {
        const long long row = j < kListSmem ? s_list[prv][j] : __ldcg(blist(prv) + j);
        unsigned long long d[NDIM + 1];  // all exchanges issued before any add
        d[NDIM] = atomicExch(dap + row, 0ull);
#pragma unroll
        for (int k = 0; k < NDIM; ++k) d[k] = atomicExch(dcs + row * NDIM + k, 0ull);
        if (d[NDIM]) atomicAdd(ap + row, d[NDIM]);
#pragma unroll
        for (int k = 0; k < NDIM; ++k)
          if (d[k]) atomicAdd(cs + row * NDIM + k, d[k]);
      }
    }
    if (EXT && !ONE && a.act_on) {
      // the copies went into the other lattice copy when they were made;
      // sites of different phases differ, so this phase's writes commute
      const unsigned np = min(s_pend[prv], (unsigned)a.pend_cap);
      const long long base = (2LL * blockIdx.x + prv) * a.pend_cap;
      uint32_t* const lat = prv ? a.lat2 : a.lat;
      uint32_t* const act = prv ? a.act2 : a.act;
      for (unsigned j = first; j < np; j += blockDim.x) {
        const uint4 e = __ldcg(a.pend + base + j);
        const unsigned long long site = (unsigned long long)e.x | ((unsigned long long)e.y << 32);
        lat[site] = e.z;
        act[site] = e.w;
      }
    }
  };

  // ---- the phase at hand: targets, tasks, draws ----------------------------------
  int cx = 0, cy = 0, cz = 0;    // the slot's parity class
  unsigned long long phase = 0;
  const int rows = a.rows;
  int nx = 0, ny = 0, nz = 1;
  unsigned r_fixed = 0;  // (batches)
  int ncx = 0, ncy = 0, tnx = 1, tny = 1, ntasks = 0;
  unsigned inv_tnx = 0;
  int task = 0, j = 0, j1 = -1;  // next target row of the task, its end (-1: no task yet)
  int x = 0, z = 0;              // the lane's column
  bool in_x = false;
  auto enter = [&]() {  // the constants of the replica in ctx
    r = ctx.rep;
    nx = ctx.nx;
    ny = ctx.ny;
    nz = NDIM == 3 ? ctx.nz : 1;
    r_fixed = ctx.fixed_mask;
  };
  auto task_grid = [&]() {
    ncx = class_count(nx, cx);
    ncy = class_count(ny, cy);
    tnx = (ncx + 31) >> 5;
    tny = (ncy + rows - 1) / rows;
    inv_tnx = task_reciprocal(tnx);
  };
  auto by_tnx = [&](const unsigned n, unsigned& rem) {
    return task_quotient(n, (unsigned)tnx, inv_tnx, rem);
  };
  auto place = [&](const int local) {  // task `local` of the lattice
    unsigned tx, turn;
    const int rest = (int)by_tnx((unsigned)local, tx);
    by_tnx((unsigned)rest, turn);
    tx += turn;
    if (tx >= (unsigned)tnx) tx -= (unsigned)tnx;
    const int tz = NDIM == 3 ? rest / tny : 0, ty = rest - tz * tny;
    j = ty * rows;
    j1 = min(ncy, j + rows);
    const int i = (int)tx * 32 + lane;
    in_x = i < ncx;
    x = in_x ? class_coord(nx, cx, i) : 0;
    z = NDIM == 3 ? class_coord(nz, cz, tz) : 0;
  };
  // KR rows of targets from row j on: their sites, their sources' sites and
  // directions, and the words for acceptance.
  uint32_t site[KR], source[KR], word[KR];
  int kd[KR];
  auto draw_rows = [&](auto&& load_target, auto&& load_source) {
    const unsigned plane = (unsigned)nx * (unsigned)ny;
    uint32_t c[KR][4];
    int ys[KR];
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      ys[u] = class_coord(ny, cy, min(j + u, j1 - 1));
      site[u] = (unsigned)z * plane + (unsigned)ys[u] * (unsigned)nx + (unsigned)x;
      load_target(u);
    }
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      c[u][0] = site[u];
      c[u][1] = (uint32_t)phase;
      c[u][2] = a.stream0 + (uint32_t)r;
      c[u][3] = (uint32_t)(phase >> 32);
      philox4x32_10(c[u][0], c[u][1], c[u][2], c[u][3], k0, k1);
    }
#pragma unroll
    for (int u = 0; u < KR; ++u) {
      kd[u] = (int)__umulhi(c[u][0], (unsigned)NB);
      int sx, sy, sz;
      source_coords<NDIM>(kd[u], x, ys[u], z, nx, ny, nz, sx, sy, sz);
      source[u] = (NDIM == 3 ? (unsigned)sz * plane : 0u) + (unsigned)sy * (unsigned)nx +
                  (unsigned)sx;
      word[u] = c[u][1];
      load_source(u);
    }
  };
  // The phase of slot `slot` at MCS `tick`, and the draws of this warp's first
  // task, in small lattices its only one.  They read no site and no table, so
  // they are made between the block's arrival at the barrier before the phase and
  // its wait, and are kept in the warp's queue, empty then: 101 x 75 x 61 box, 20
  // MCS 2.78 -> 2.51 ms; 1001 x 777, 20 MCS 0.98 -> 0.86; 96^3 with persistence
  // 1.46 -> 1.33; act on 512^2, 50 MCS 1.90 -> 1.80; 4096^2, 50 MCS 6.97 -> 6.70;
  // 256^3, 20 MCS 3.54 -> 3.28; batches of 16 x 64^2, 20 MCS 0.463 -> 0.444, of 32
  // x 128^2 0.661 -> 0.613, large ones the same.  (Held in registers they made
  // every kernel spill: 4096^2 7.80.)  Not in batches with scores, which it makes
  // spill (gradient of 128 x 256^2 24.1 -> 24.4 ms).
  constexpr bool AHEAD = !(BATCH && SCORE);
  bool drawn = false;
  int first = 0;             // (batches) first task of the replica at hand
  auto replica_of = [&](const int t) {
    // the largest with pre[lo] <= t (tasks of the slot before each replica),
    // 32 probes at a time
    const int* pre = a.task_prefix + (cx + 3 * cy + 9 * cz) * (a.nrep + 1);
    int lo = 0, n = a.nrep;
    while (n > 1) {
      const int st = (n + 31) >> 5, k = lane * st;
      const int v = k < n ? __ldg(pre + lo + k) : 0;
      const int at = __popc(__ballot_sync(kFull, k < n && v <= t)) - 1;
      first = __shfl_sync(kFull, v, at);
      lo += at * st;
      n = min(st, n - at * st);
    }
    return a.rep_map ? __ldg(a.rep_map + lo) : lo;
  };
  auto switch_to = [&](const int rep) {
    flush_counters();
    __syncwarp();
    load_replica(rep);
    __syncwarp();
    enter();
  };
  auto begin_phase = [&](const int slot, const unsigned long long tick, const int b, const int G) {
    cx = slot % 3, cy = (slot / 3) % 3, cz = slot / 9;
    phase = tick * NSLOTS + (unsigned long long)slot;
    task = b + warp * G;
    j = 0, j1 = -1;
    x = z = 0;
    in_x = false;
    if constexpr (BATCH) {
      ntasks = __ldg(a.task_prefix + slot * (a.nrep + 1) + a.nrep);
    } else {
      enter();
      task_grid();
      ntasks = tnx * tny * class_count(nz, cz);
    }
    if constexpr (AHEAD) drawn = task < ntasks;
    if (AHEAD && drawn) {
      if constexpr (BATCH) {
        const int rep = replica_of(task);
        if (rep != r) switch_to(rep);
        task_grid();
      }
      place(task - first);
      draw_rows([](int) {}, [](int) {});
      uint4* const q = reinterpret_cast<uint4*>(queue);
#pragma unroll
      for (int u = 0; u < KR; ++u)
        q[32 * u + lane] = make_uint4(site[u], source[u], word[u], (uint32_t)kd[u]);
    }
  };

  // ---- one phase ----------------------------------------------------------------
  // G blocks share the slot's tasks, this one is number b.
  auto run_phase = [&](const int slot, const unsigned long long tick, const int step, const int b,
                       const int G) {
    const int cur = step & 1;
    PhaseTables<NDIM> held;
    if constexpr (!SHARED_PT) held = tables_of(cur);
    const PhaseTables<NDIM>& pt = SHARED_PT ? s_pt[cur] : held;
    // the lattice (act stamps) the phase reads, and the one it writes:
    // another copy in act runs that have one
    const bool two = EXT && !ONE && a.act_on;
    const uint32_t* const lat_r = two && cur ? a.lat2 : a.lat;
    uint32_t* const lat_w = two && !cur ? a.lat2 : a.lat;
    const uint32_t* const act_r = !ONE && cur ? a.act2 : a.act;
    uint32_t* const act_w = cur ? a.act : a.act2;  // (not in ONE)

    // Changed rows (0xFFFFFFFF: none) of the lanes onto the block's dirty list:
    // one shared-memory atomic per batch.
    auto push_rows = [&](const unsigned push_s, const unsigned push_t) {
      const unsigned bs = __ballot_sync(kFull, push_s != 0xFFFFFFFFu);
      const unsigned bt = __ballot_sync(kFull, push_t != 0xFFFFFFFFu);
      if ((bs | bt) && !a.scan) {  // warp-uniform
        const unsigned npush = (unsigned)(__popc(bs) + __popc(bt));
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&s_cnt[cur], npush);
        at = __shfl_sync(kFull, at, 0);
        // The host sizes the lists for two rows per attempt; a list that
        // would still overflow is reported, never written past its end.
        if ((long long)at + npush > a.list_cap) {
          if (lane == 0) atomicOr(err, kErrListFull);
        } else {
          auto put = [&](unsigned i, unsigned row) {
            if (i < kListSmem)
              s_list[cur][i] = row;
            else
              blist(cur)[i] = row;
          };
          if (push_s != 0xFFFFFFFFu) put(at + __popc(bs & lanemask_lt()), push_s);
          if (push_t != 0xFFFFFFFFu) put(at + __popc(bs) + __popc(bt & lanemask_lt()), push_t);
        }
      }
    };

    // ---- evaluate: n <= 32 attempts, one per lane -------------------------------
    auto evaluate = [&](const Attempt* q, const int n) {
      const uint32_t* const L = lat_r + ctx.lat_off;
      bool accepted = false;
      unsigned push_s = 0xFFFFFFFFu, push_t = 0xFFFFFFFFu;  // table rows this lane changed
      uint32_t at_site = 0, area_s = 0, area_t = 0, change = 0;  // (DEFER)
      if (lane < n) {
        const uint4 e = *reinterpret_cast<const uint4*>(q + lane);
        const uint32_t site = e.x, s = e.z, t = e.w;
        const uint32_t is = s & 0xFFFFFFu, it = t & 0xFFFFFFu;
        if (max(is, it) > (uint32_t)ctx.ncells) {
          atomicOr(err, kErrBadId);
        } else {
          const int kdir = (int)(e.y & 0xFFu);
          const int ts = (int)(s >> 24) & (kMaxTypes - 1);
          const int tt = (int)(t >> 24) & (kMaxTypes - 1);
          const unsigned rs = (unsigned)ctx.cell_off + is, rt = (unsigned)ctx.cell_off + it;
          // (the medium's row exists; its values are not used)
          const unsigned long long aps = __ldcg(pt.rap + rs), apt = __ldcg(pt.rap + rt);
          // centroid sums, needed only on acceptance: fetched with the row
          // where many attempts are accepted and registers allow (batches,
          // scores: 256 ragged replicas 17.4 ms, on acceptance 18.1)
          constexpr bool kEarlyCs = NDIM == 2 && (BATCH || MODE != kPlain);
          long long cs_s[NDIM], cs_t[NDIM];
          if constexpr (kEarlyCs) {
            const longlong2 vs = __ldcg(reinterpret_cast<const longlong2*>(pt.rcs) + rs);
            const longlong2 vt = __ldcg(reinterpret_cast<const longlong2*>(pt.rcs) + rt);
            cs_s[0] = vs.x, cs_s[1] = vs.y, cs_t[0] = vt.x, cs_t[1] = vt.y;
          }
          const DevParams* const P = ctx.P;
          const int nx = ctx.nx, ny = ctx.ny, nz = NDIM == 3 ? ctx.nz : 1;
          const unsigned plane = (unsigned)nx * (unsigned)ny;
          const int z = NDIM == 3 ? (int)fast_div(site, ctx.div_plane) : 0;
          const unsigned in_plane = NDIM == 3 ? site - (unsigned)z * plane : site;
          const int y = (int)fast_div(in_plane, ctx.div_nx),
                    x = (int)(in_plane - (unsigned)y * nx);
          // offsets of the neighbouring columns, rows and planes (wrapped)
          const int xl = x ? -1 : nx - 1, xr = x + 1 < nx ? 1 : 1 - nx;
          const int yl = y ? -nx : (int)plane - nx, yr = y + 1 < ny ? nx : nx - (int)plane;
          const int zl = NDIM == 3 ? (z ? -(int)plane : (nz - 1) * (int)plane) : 0;
          const int zr = NDIM == 3 ? (z + 1 < nz ? (int)plane : -(nz - 1) * (int)plane) : 0;
          uint32_t nb[NBC];
#pragma unroll
          for (int p = 0; p < (NDIM == 3 ? 3 : 1); ++p)
#pragma unroll
            for (int m = 0; m < 3; ++m) {
              const uint32_t* c = L + site + (NDIM == 3 ? (p == 0 ? zl : p == 1 ? 0 : zr) : 0) +
                                  (m == 0 ? yl : m == 1 ? 0 : yr);
              nb[9 * p + 3 * m] = c[xl];
              nb[9 * p + 3 * m + 1] = c[0];
              nb[9 * p + 3 * m + 2] = c[xr];
            }
          // Adhesion of both configurations, summed in neighbour order.  Every
          // value is loaded, so that no load waits on a comparison.
          float e_old = 0.0f, e_new = 0.0f;
          int cnt_s = 0, cnt_t = 0;
          unsigned by_new = 0, by_old = 0;  // (scores) neighbours by type, a byte each
          auto adhesion = [&](const float* Jt, const float* Js, auto&& load) {
#pragma unroll
            for (int k = 0; k < NBC; ++k) {
              if (k == NB / 2) continue;  // the target itself
              const uint32_t v = nb[k];
              const int tn = (int)(v >> 24) & (kMaxTypes - 1);
              const float jt = load(Jt + tn), js = load(Js + tn);
              const bool is_t = v == t, is_s = v == s;
              e_old = is_t ? e_old : __fadd_rn(e_old, jt);
              e_new = is_s ? e_new : __fadd_rn(e_new, js);
              cnt_t += is_t;
              cnt_s += is_s;
              if (SCORE && tn < kScoreTypes) {
                by_new += is_s ? 0u : 1u << (8 * tn);
                by_old += is_t ? 0u : 1u << (8 * tn);
              }
            }
          };
          if constexpr (BATCH)
            adhesion(P->J + tt * kMaxTypes, P->J + ts * kMaxTypes,
                     [](const float* p) { return __ldg(p); });
          else
            adhesion(s_J + tt * kJPitch, s_J + ts * kJPitch, [](const float* p) { return *p; });
          if (ctx.stick_on) {
            // stickiness of the old configuration, summed in neighbour order
            // and added to its adhesion as one term (neighbours read again:
            // kept past the adhesion sums they cost the other runs spills)
            float e_st = 0.0f;
            const float* St = P->stick + tt * kMaxTypes;
#pragma unroll 1
            for (int p = 0; p < (NDIM == 3 ? 3 : 1); ++p)
#pragma unroll 1
              for (int m = 0; m < 3; ++m) {
                const uint32_t* c = L + site + (NDIM == 3 ? (p == 0 ? zl : p == 1 ? 0 : zr) : 0) +
                                    (m == 0 ? yl : m == 1 ? 0 : yr);
                const uint32_t v3[3] = {c[xl], c[0], c[xr]};
#pragma unroll
                for (int k = 0; k < 3; ++k)  // (the target itself holds t)
                  if (v3[k] != t)
                    e_st = __fadd_rn(e_st, __ldg(St + ((int)(v3[k] >> 24) & (kMaxTypes - 1))));
              }
            e_old = __fadd_rn(e_old, e_st);
          }
          float dH = __fsub_rn(e_new, e_old);
          {
            // chemotaxis first, as in the reference's sum; lambda of the
            // source type, of the target type for a medium source
            float chemo = 0.0f;
            if (ctx.chemo_on) {
              const float lam = __ldg(&P->chemo[ts ? ts : tt]);
              if (lam != 0.0f)
                chemo = __fmul_rn(-lam, chemo_dot<NDIM>(a.field + NDIM * ctx.lat_off,
                                                        (long long)plane * nz, x, y, z, kdir, nx,
                                                        ny, nz));
            }
            // persistence next (3D): lambda of the source type (target type for
            // a medium source), preferred direction of the source cell (of the
            // target cell for a medium source), src/kernels3d.cu:327-343
            if (EXT && NDIM == 3 && ctx.persist_on) {
              const float lam = __ldg(&P->persist_lambda[ts ? ts : tt]);
              if (lam != 0.0f) {
                float ux, uy, uz;
                int sx, sy, sz;
                unit_dir<NDIM>(kdir, x, y, z, nx, ny, nz, ux, uy, uz, sx, sy, sz);
                const double* pd = a.prefdir + 3LL * (is ? rs : rt);
                float c = __fmul_rn(ux, (float)__ldg(pd));
                c = __fmaf_rn(uy, (float)__ldg(pd + 1), c);
                c = __fmaf_rn(uz, (float)__ldg(pd + 2), c);
                chemo = __fadd_rn(chemo, __fmul_rn(-lam, c));
              }
            }
            // act next: lambda and max of the target type, of the source type
            // for a medium target
            if (EXT && ctx.act_on) {
              const int ta = tt ? tt : ts;
              const float lam = __ldg(&P->act_lambda[ta]);
              const int amax_a = __ldg(&P->act_max[ta]);
              if (lam != 0.0f && amax_a != 0) {
                int sx, sy, sz;
                source_coords<NDIM>(kdir, x, y, z, nx, ny, nz, sx, sy, sz);
                const long long tk = (long long)tick;
                const uint32_t* const A = act_r + ctx.lat_off;
                const float tgt = t ? act_mean<NDIM>(L, A, x, y, z, nx, ny, nz, t,
                                                     __ldg(&P->act_max[tt]), tk)
                                    : 0.0f;
                const float src = s ? act_mean<NDIM>(L, A, sx, sy, sz, nx, ny, nz, s,
                                                     __ldg(&P->act_max[ts]), tk)
                                    : 0.0f;
                chemo = __fadd_rn(chemo, __fmul_rn(__fdiv_rn(-lam, (float)amax_a),
                                                   __fsub_rn(src, tgt)));
              }
            }
            dH = __fadd_rn(chemo, dH);
          }
          const int dps = NB - 2 * cnt_s;
          const int dpt = 2 * cnt_t - NB;
          TypeParams ps, pr;
          if constexpr (BATCH) {
            ps = {__ldg(&P->lam_area[ts]), __ldg(&P->tgt_area[ts]), __ldg(&P->lam_perim[ts]),
                  __ldg(&P->tgt_perim[ts])};
            pr = {__ldg(&P->lam_area[tt]), __ldg(&P->tgt_area[tt]), __ldg(&P->lam_perim[tt]),
                  __ldg(&P->tgt_perim[tt])};
          } else {
            ps = s_type[ts];
            pr = s_type[tt];
          }
          float qps, qpt, qas, qat;
          // (scores) the same of the whole copy.  As sums of exact FP32 integers
          // and of 32-bit ones where those do: in 64 bits, or chosen beside the
          // scores, gradients of 128 x 256^2 took 24.3 to 24.5 ms, so 23.9.
          float q_area = 0.0f, q_perim = 0.0f;
          const int As = unpack_area(aps), At = unpack_area(apt);
          const int Ps = unpack_perim(aps), Pt = unpack_perim(apt);
          if (ctx.small_targets && (unsigned)(As | At | Ps | Pt) < kSmallTable) {
            constraint_terms_small(As, Ps, dps, 1, ps, qps, qas);
            constraint_terms_small(At, Pt, dpt, -1, pr, qpt, qat);
            if constexpr (SCORE) {
              q_area = (s ? qas : 0.0f) + (t ? qat : 0.0f);
              if (a.score_spec.lambda_perim)
                q_perim = (float)((s ? dps * (2 * (Ps - ps.tgt_perim) + dps) : 0) +
                                  (t ? dpt * (2 * (Pt - pr.tgt_perim) + dpt) : 0));
            }
          } else {
            constraint_terms_wide(As, Ps, dps, 1, ps, qps, qas);
            constraint_terms_wide(At, Pt, dpt, -1, pr, qpt, qat);
            if constexpr (SCORE) {
              q_area = __ll2float_rn((s ? 1 + 2 * ((long long)As - ps.tgt_area) : 0LL) +
                                     (t ? 1 - 2 * ((long long)At - pr.tgt_area) : 0LL));
              q_perim = __ll2float_rn(
                  (s ? dps * (2 * ((long long)Ps - ps.tgt_perim) + dps) : 0LL) +
                  (t ? dpt * (2 * ((long long)Pt - pr.tgt_perim) + dpt) : 0LL));
            }
          }
          if (ctx.perim_on) {
            dH = s ? __fmaf_rn(ps.lam_perim, qps, dH) : dH;
            dH = t ? __fmaf_rn(pr.lam_perim, qpt, dH) : dH;
          }
          dH = s ? __fmaf_rn(ps.lam_area, qas, dH) : dH;
          dH = t ? __fmaf_rn(pr.lam_area, qat, dH) : dH;
          const float T = ctx.temperature;
          float ex = 1.0f;  // exp(-dH/T) when 0 <= dH and T > 0
          const bool ok = metropolis(dH, T, e.y, ex);
          if (SCORE && dH >= 0.0f && T > 0.0f) {
            // d log P(decision) / d theta with P(accept) = min(1, exp(-dH/T)):
            // accept: -g, reject: e/(1-e) g, g = d(dH/T)/d theta.  At
            // dH = 0 exactly (integer parameters make it common) P has a
            // kink, slope -g on one side and 0 on the other; the score takes
            // the mean of the two one-sided derivatives, -g/2.
            const float xT = dH / T;
            const float om = xT < 1e-2f
                                 ? xT * (1.0f - 0.5f * xT * (1.0f - (xT / 3.0f) *
                                                                        (1.0f - 0.25f * xT)))
                                 : 1.0f - ex;  // 1 - exp(-x)
            const float cT = (dH == 0.0f ? -0.5f : (ok ? -1.0f : ex / om)) / T;
#pragma unroll
            for (int p = 0; p < kScorePairsMax; ++p) {
              if (p < a.score_spec.n_pairs) {
                const int pa = a.score_spec.pair_a[p], pb = a.score_spec.pair_b[p];
                int d = 0;
                if (ts == pa) d += (by_new >> (8 * pb)) & 0xFF;
                if (pa != pb && ts == pb) d += (by_new >> (8 * pa)) & 0xFF;
                if (tt == pa) d -= (by_old >> (8 * pb)) & 0xFF;
                if (pa != pb && tt == pb) d -= (by_old >> (8 * pa)) & 0xFF;
                sc[p] += cT * (float)d;
              }
            }
            if (a.score_spec.lambda_area) sc[kScorePairsMax] += cT * q_area;
            if (a.score_spec.lambda_perim) sc[kScorePairsMax + 1] += cT * q_perim;
            if (a.score_spec.temperature) sc[kScorePairsMax + 2] -= cT * xT;
          }
          if (ok) {
            accepted = true;
            if constexpr (!ONE) lat_w[ctx.lat_off + site] = s;
            if (EXT && a.act_on) {  // into this copy in the next phase (ONE: after this one)
              if constexpr (!ONE) act_w[ctx.lat_off + site] = (uint32_t)tick;
              const unsigned j = atomicAdd(&s_pend[cur], 1u);
              if ((long long)j < a.pend_cap) {
                const unsigned long long g = (unsigned long long)ctx.lat_off + site;
                if constexpr (ONE) {
                  pend_site(a, j) = g;
                  pend_value(a, j) = s;
                } else {
                  a.pend[(2LL * blockIdx.x + cur) * a.pend_cap + j] =
                      make_uint4((uint32_t)g, (uint32_t)(g >> 32), s, (uint32_t)tick);
                }
              } else {
                atomicOr(err, kErrListFull);  // reported, never written past the end
              }
            }
            if constexpr (DEFER) {
              if (s) push_s = rs;
              if (t) push_t = rt;
              area_s = (uint32_t)As, area_t = (uint32_t)At;
              at_site = site;
              change = (uint32_t)(dps + 64) | ((uint32_t)(dpt + 64) << 16);
            } else {
              const int crd[3] = {x, y, z};
              const int dim[3] = {nx, ny, nz};
              long long img[NDIM];
              if (s) {
    #pragma unroll
                for (int k = 0; k < NDIM; ++k)
                  img[k] = nearest_image(
                      crd[k], dim[k], As,
                      kEarlyCs ? cs_s[k] : __ldcg(pt.rcs + (long long)rs * NDIM + k));
                add_delta<NDIM>(pt, rs, 1, dps, img, 1);
                push_s = rs;
              }
              if (t) {
    #pragma unroll
                for (int k = 0; k < NDIM; ++k)
                  img[k] = nearest_image(
                      crd[k], dim[k], At,
                      kEarlyCs ? cs_t[k] : __ldcg(pt.rcs + (long long)rt * NDIM + k));
                add_delta<NDIM>(pt, rt, -1, dpt, img, -1);
                push_t = rt;
              }
            }
          }
        }
      }
      if constexpr (DEFER) {
        const unsigned bs = __ballot_sync(kFull, push_s != 0xFFFFFFFFu);
        const unsigned bt = __ballot_sync(kFull, push_t != 0xFFFFFFFFu);
        uint4* const q = reinterpret_cast<uint4*>(changes) + nchange;
        if (push_s != 0xFFFFFFFFu)
          q[__popc(bs & lanemask_lt())] = make_uint4(push_s, at_site, area_s, change & 0xFFFFu);
        if (push_t != 0xFFFFFFFFu)
          q[__popc(bs) + __popc(bt & lanemask_lt())] =
              make_uint4(push_t, at_site, area_t, (change >> 16) | 256u);
        nchange += __popc(bs) + __popc(bt);
      }
      n_acc += __popc(__ballot_sync(kFull, accepted));
      if constexpr (!DEFER) push_rows(push_s, push_t);
    };

    // ---- n <= 32 queued row changes, one per lane ------------------------------
    auto change_rows = [&](const RowChange* q, const int n) {
      unsigned row = 0xFFFFFFFFu;
      if (lane < n) {
        const uint4 e = *reinterpret_cast<const uint4*>(q + lane);
        row = e.x;
        const int lost = (int)(e.w >> 8), area = (int)e.z;
        const unsigned site = e.y;
        const int nx = ctx.nx, ny = ctx.ny, nz = NDIM == 3 ? ctx.nz : 1;
        const int z = NDIM == 3 ? (int)fast_div(site, ctx.div_plane) : 0;
        const unsigned in_plane =
            NDIM == 3 ? site - (unsigned)z * ((unsigned)nx * (unsigned)ny) : site;
        const int y = (int)fast_div(in_plane, ctx.div_nx), x = (int)(in_plane - (unsigned)y * nx);
        const int crd[3] = {x, y, z};
        const int dim[3] = {nx, ny, nz};
        long long cs[NDIM], img[NDIM];
        if constexpr (NDIM == 2) {
          const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(pt.rcs) + row);
          cs[0] = v.x, cs[1] = v.y;
        } else {
#pragma unroll
          for (int k = 0; k < NDIM; ++k) cs[k] = __ldcg(pt.rcs + (long long)row * NDIM + k);
        }
#pragma unroll
        for (int k = 0; k < NDIM; ++k) img[k] = nearest_image(crd[k], dim[k], area, cs[k]);
        add_delta<NDIM>(pt, row, lost ? -1 : 1, (int)(e.w & 0xFFu) - 64, img, lost ? -1 : 1);
      }
      push_rows(row, 0xFFFFFFFFu);
    };

    auto flush_changes = [&](const int least) {  // while at least that many are queued
      while (nchange >= least) {
        const int n = min(32, nchange);
        nchange -= n;
        change_rows(changes + nchange, n);
        __syncwarp();
      }
    };

    const uint32_t* L = lat_r + (!BATCH || r >= 0 ? ctx.lat_off : 0);
    unsigned* ctr = &s_next[step & 1];
    if (tid == 0) s_next[(step + 1) & 1] = 0u;
    int nq = 0;
    int next_rep = -1;      // (batches) the replica of the task at hand
    bool rep_ready = true;  // its constants are loaded
    int pool_at = -1, pool_n = 0;  // pooled stage: this warp's next batch, all attempts
    for (;;) {
      const Attempt* batch = queue;
      int nbatch = 0;
      while (pool_at < 0) {
        if (nq >= 32) {  // the last 32
          nq -= 32;
          batch = queue + nq;
          nbatch = 32;
          break;
        }
        if (j >= j1) {  // the next task
          if (j1 >= 0) {
            unsigned v = 0;
            if (lane == 0) v = atomicAdd(ctr, 1u);
            task = b + (wpb + (int)__shfl_sync(kFull, v, 0)) * G;
          }
          j = 0;
          j1 = 0;
          if (task >= ntasks) {
            if constexpr (BATCH) {  // what is left of the warp's last replica
              pool_at = 0;
              pool_n = nq;
              break;
            }
            unsigned at = 0;
            if (lane == 0 && nq) at = atomicAdd(&s_pool, (unsigned)nq);
            at = __shfl_sync(kFull, at, 0);
            if (lane < nq)
              *reinterpret_cast<uint4*>(pool + at + lane) =
                  *reinterpret_cast<const uint4*>(queue + lane);
            __syncthreads();
            pool_n = (int)s_pool;
            pool_at = warp * 32;
            break;
          }
          if constexpr (BATCH) {
            next_rep = replica_of(task);
            rep_ready = false;
            j1 = 1;  // a task is at hand
          }
        }
        if constexpr (BATCH) {
          if (!rep_ready) {
            if (next_rep != r) {
              if (nq > 0) {  // the last replica's attempts first
                nbatch = nq;
                nq = 0;
                break;
              }
              if constexpr (DEFER) flush_changes(1);
              if (SCORE && r >= 0) flush_scores(a, sc, r, tick);
              switch_to(next_rep);
              L = lat_r + ctx.lat_off;
            }
            task_grid();
            rep_ready = true;
            j1 = 0;
          }
        }
        if (j1 == 0) place(task - first);
        uint32_t tv[KR], sv[KR];
        const unsigned fixed_mask = BATCH ? r_fixed : ctx.fixed_mask;
        if (AHEAD && drawn) {
          drawn = false;
          const uint4* const q = reinterpret_cast<const uint4*>(queue);
#pragma unroll
          for (int u = 0; u < KR; ++u) {
            const uint4 e = q[32 * u + lane];
            site[u] = e.x, source[u] = e.y, word[u] = e.z, kd[u] = (int)e.w;
          }
          __syncwarp();  // the queue is written next
#pragma unroll
          for (int u = 0; u < KR; ++u) tv[u] = L[site[u]], sv[u] = L[source[u]];
        } else {
          draw_rows([&](int u) { tv[u] = L[site[u]]; }, [&](int u) { sv[u] = L[source[u]]; });
        }
#pragma unroll
        for (int u = 0; u < KR; ++u) {
          uint32_t s = sv[u];
          bool keep = in_x && j + u < j1 && s != tv[u];
          if (fixed_mask && keep) {
            // a target of a fixed type never changes; a source of a fixed type
            // proposes the medium instead (src/kernels2d.cu:280-290)
            if ((fixed_mask >> ((tv[u] >> 24) & (kMaxTypes - 1))) & 1u) {
              keep = false;
            } else if ((fixed_mask >> ((s >> 24) & (kMaxTypes - 1))) & 1u) {
              s = 0u;
              keep = tv[u] != 0u;
            }
          }
          const unsigned ball = __ballot_sync(kFull, keep);
          if (keep)
            *reinterpret_cast<uint4*>(queue + nq + __popc(ball & lanemask_lt())) =
                make_uint4(site[u], (word[u] & 0xFFFFFF00u) | (uint32_t)kd[u], s, tv[u]);
          nq += __popc(ball);
          n_eval += __popc(ball);
        }
        j += KR;
        __syncwarp();
      }
      if (pool_at >= 0) {
        if (pool_at >= pool_n) break;
        batch = (BATCH ? queue : pool) + pool_at;
        nbatch = min(32, pool_n - pool_at);
        pool_at += BATCH ? pool_n : wpb * 32;
      }
      evaluate(batch, nbatch);
      __syncwarp();  // the queue is rewritten next
      if constexpr (DEFER) flush_changes(32);
    }
    if constexpr (DEFER) flush_changes(1);
    if (SCORE && BATCH && r >= 0) flush_scores(a, sc, r, tick);
  };

  // All MCS of the launch over the lattice or batch (this block is number b
  // of G), or over each replica that this block claims (G = 1; block barriers
  // between its phases).  The first grid barrier of replica dispatch makes
  // every block read the starting tick before block 0 can advance it.
  const bool local = !BATCH && a.block_local;
  const int G = local ? 1 : (int)gridDim.x, b = local ? 0 : (int)blockIdx.x;
  if (local && !grid_barrier(a.ctl, ++episode, &s_ok)) return;
  for (;;) {
    if constexpr (!BATCH) {
      if (warp == 0) {
        int qi = 0;
        if (local && lane == 0) qi = (int)atomicAdd(&a.ctl[kCtlQueue], 1u);
        qi = __shfl_sync(kFull, qi, 0);
        if (lane == 0) s_claim = qi;
        if (!local || qi < a.queue_len) load_replica(local ? __ldg(a.rep_order + qi) : 0);
      }
      __syncthreads();
      if (local && s_claim >= a.queue_len) break;  // block-uniform
      const DevParams* const P = ctx.P;
      for (int i = tid; i < kMaxTypes * kMaxTypes; i += blockDim.x)
        s_J[(i / kMaxTypes) * kJPitch + i % kMaxTypes] = __ldg(&P->J[i]);
      for (int i = tid; i < kMaxTypes; i += blockDim.x)
        s_type[i] = {__ldg(&P->lam_area[i]), __ldg(&P->tgt_area[i]), __ldg(&P->lam_perim[i]),
                     __ldg(&P->tgt_perim[i])};
      __syncthreads();
    }
    int step = 0;
    if (a.mcs > 0) begin_phase(a.slots[0], s_tick0, b, G);
    for (int m = 0; m < a.mcs; ++m) {
      const unsigned long long tick = s_tick0 + (unsigned long long)m;
      for (int si = 0; si < a.nslot_active; ++si, ++step) {
        const int prv = (step & 1) ^ 1;
        // from the last thread down: the first warps have the first tasks
        if (step > 0) replay_phase(prv, blockDim.x - 1 - tid);
        run_phase(a.slots[si], tick, step, b, G);
        __syncthreads();
        if constexpr (ONE) {
          // the phase's copies are made when all its attempts are
          if (!local && !grid_barrier(a.ctl, ++episode, &s_ok)) return;
          const unsigned np = min(s_pend[step & 1], (unsigned)a.pend_cap);
          for (unsigned j = tid; j < np; j += blockDim.x) {
            const unsigned long long site = pend_site(a, j);
            a.lat[site] = pend_value(a, j);
            a.act[site] = (uint32_t)tick;
          }
          __syncthreads();
        }
        if (tid == 0) {
          s_cnt[prv] = s_pend[prv] = 0;
          s_pool = 0;
          if (!local) grid_arrive(a.ctl);
        }
        const bool wrap = si + 1 == a.nslot_active;
        if (!wrap || m + 1 < a.mcs)
          begin_phase(a.slots[wrap ? 0 : si + 1], tick + (wrap ? 1 : 0), b, G);
        if (local)
          __syncthreads();
        else if (!grid_wait(a.ctl, ++episode, &s_ok))
          return;
      }
      if (SCORE && !BATCH) flush_scores(a, sc, r, tick);
      if (n_eval > (1u << 30)) flush_counters();  // (a phase adds less than 2^31)
    }
    // Final replay: the last phase's deltas into the copy it read, so that
    // both copies agree when the launch ends.
    if (step > 0) replay_phase((step - 1) & 1, tid);
    flush_counters();
    if (!local) break;
    __syncthreads();
    if (tid < 2) s_cnt[tid] = s_next[tid] = s_pend[tid] = 0;
    __syncthreads();
  }
  if (a.tick_ptr && a.tick_advance && blockIdx.x == 0 && tid == 0 && a.mcs > 0)
    *a.tick_ptr = s_tick0 + (unsigned long long)a.mcs;
}

template <int NDIM, int KR, int MODE, bool BATCH, bool LOCAL>
struct SweepFn {
  static const void* fn() { return (const void*)sweep_kernel<NDIM, KR, MODE, BATCH, LOCAL>; }
  static size_t smem(int warps) { return (size_t)warps * warp_smem<NDIM, KR, MODE, BATCH>(); }
};

template <int NDIM, int KR, int MODE, bool BATCH, bool LOCAL = false>
cudaError_t launch_sweep_as(const SweepArgs& a, int grid, int warps, cudaStream_t s) {
  using F = SweepFn<NDIM, KR, MODE, BATCH, LOCAL>;
  constexpr int kMaxWarps = sweep_warps<NDIM, KR, MODE, BATCH>();
  const int w = warps < kMaxWarps ? warps : kMaxWarps;
  // The limit belongs to the function on the device: every launch sets the
  // same one, whatever its own size, so that a launch of another engine in
  // another thread cannot lower it in between.
  const cudaError_t e = cudaFuncSetAttribute(
      F::fn(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::smem(kMaxWarps));
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<SweepArgs*>(&a)};
  return cudaLaunchCooperativeKernel(F::fn(), dim3(grid), dim3(32 * w), args, F::smem(w), s);
}

// One kernel per mode and rows drawn side by side (a.kr): one, three or four;
// in batches two, and four where tasks have as many rows (more loads in
// flight: 256 ragged replicas, 20 MCS 17.4 / 16.8 ms, gradient of 128 x 256^2
// 24.8 / 24.3); two in the extended and single-lattice score kernels.
template <int NDIM>
cudaError_t launch_sweep_nd(const SweepArgs& a, bool batch, bool scores, int grid, int warps,
                            cudaStream_t s) {
  const bool ext = a.act_on || a.prefdir, one = a.act_on && !a.lat2;
  if (batch) {
    if (one) return launch_sweep_as<NDIM, 2, kOne, true>(a, grid, warps, s);
    if (ext) return launch_sweep_as<NDIM, 2, kExt, true>(a, grid, warps, s);
    if constexpr (NDIM == 2) {
      if (scores)
        return a.kr == 4 ? launch_sweep_as<NDIM, 4, kScore, true>(a, grid, warps, s)
                         : launch_sweep_as<NDIM, 2, kScore, true>(a, grid, warps, s);
    }
    return a.kr == 4 ? launch_sweep_as<NDIM, 4, kPlain, true>(a, grid, warps, s)
                     : launch_sweep_as<NDIM, 2, kPlain, true>(a, grid, warps, s);
  }
  if (one) return launch_sweep_as<NDIM, 2, kOne, false>(a, grid, warps, s);
  if (ext) return launch_sweep_as<NDIM, 2, kExt, false>(a, grid, warps, s);
  if constexpr (NDIM == 2) {
    if (scores) return launch_sweep_as<NDIM, 2, kScore, false>(a, grid, warps, s);
  }
  switch (a.kr) {
    case 1: return launch_sweep_as<NDIM, 1, kPlain, false>(a, grid, warps, s);
    case 4:
      if (NDIM == 2 && a.block_local)
        return launch_sweep_as<NDIM, 4, kPlain, false, NDIM == 2>(a, grid, warps, s);
      return launch_sweep_as<NDIM, 4, kPlain, false>(a, grid, warps, s);
    default: return launch_sweep_as<NDIM, 3, kPlain, false>(a, grid, warps, s);
  }
}

}  // namespace
}  // namespace gpucpm
