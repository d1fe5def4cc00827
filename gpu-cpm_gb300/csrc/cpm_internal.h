// cpm_internal.h — structures shared by the host engine (cpm_engine.cu) and
// the sm_103a kernels (cpm_kernels.cu).  Not part of the public C-ABI.
//
// Device memory layout of one engine (a batch of R replicas; a plain
// gpucpm.Cpm is a batch of one):
//   lat    : uint32 [sum_r sites_r]      replica r at reps[r].lat_off,
//                                        row-major (z*ny + y)*nx + x
//   ap[2]  : uint64 [rows]               packed (area | perimeter << 32) of
//                                        replica r's id c at row
//                                        reps[r].cell_off + c; two copies
//   cs[2]  : int64  [rows * ndim]        exact centroid coordinate sums,
//                                        two copies
//   dap[2], dcs[2]                       deltas of one phase (two phases in
//                                        flight alternate)
//   dlist  : uint32 [grid * 2 * list_cap] two dirty lists per sweep block:
//                                        rows changed in a phase (a row may
//                                        appear more than once); used where
//                                        rows are many (SweepArgs::scan)
//   ctl    : uint32 [64]                 barrier counter, replica queue,
//                                        sticky error bits
//   (optional) field (chemotaxis, float), act stamps (uint32 per site),
//   prefdir [rows][3] and the persistence ring [history][rows][3] (double)
// Table double buffering: phase k reads copy k % 2 and adds its deltas both
// into the other copy and into dap/dcs[k % 2]; phase k + 1 replays those
// deltas into copy k % 2, which missed them (every row looked at by one thread,
// or each delta of a listed row taken with an exchange, so that a row listed
// twice is replayed once).  So every phase reads
// tables as they stood when it began, with one grid barrier per phase.  The
// tables are
// small next to the lattice (4096^2 at 100 sites per cell: 67 MB of lattice,
// 4 MB per table copy) and stay L2-resident through a run.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

namespace gpucpm {

constexpr int kMaxTypes = 32;
constexpr int kSweepSmemMax = 227 * 1024;  // usable shared memory per block
constexpr int kInitThreads = 256;

// How the slots of a sweep are cut into warp tasks of 32 target columns x
// `rows` target rows, `kr` of them drawn side by side.  The sweep's result
// does not depend on it.  Four variants; the autotuner (cpm_autotune) picks
// one per engine.  Variant 0 follows from the size (plan_sweep, batch_rows),
// 1 has 8-row tasks, 2 16-row tasks, 3 one-row tasks (batches
// 8, 32 and 2).
constexpr int kTileVariants = 4;
struct SweepPlan {
  int kr, rows;
  int warps;           // per block
  int grid;            // blocks
  long long list_cap;  // dirty-list entries of a block and phase
};
// One lattice over the whole grid.  wide: the extended and score kernels
// (20 warps per block, two rows side by side).
SweepPlan plan_sweep(int ndim, int nx, int ny, int nz, int variant, int sms, bool wide);
// Rows of a batch's tasks (grid dispatch), total_units = 32-column rows of
// the largest slot.
int batch_rows(int variant, long long total_units, int sms);

// ctl[] word indices (the barrier counter has a 128-byte line of its own)
constexpr int kCtlBarrier = 0;
constexpr int kCtlQueue = 40;  // next replica to claim (replica dispatch)
constexpr int kCtlErr = 48;  // words [0, kCtlErr) are zeroed before a launch
constexpr int kCtlWords = 64;

// error bits in ctl[kCtlErr]
constexpr int kErrTimeout = 1;      // a grid barrier waited too long
constexpr int kErrBadId = 2;        // site id above the replica's ncells
constexpr int kErrBadType = 4;      // type >= kMaxTypes
constexpr int kErrMediumType = 8;   // id 0 with a non-zero type
constexpr int kErrTypeConflict = 16;  // one id with two types
constexpr int kErrListFull = 32;      // a dirty list would overflow (not written)

// Per-replica parameters, kept in global memory (read through the
// read-only cache; a replica's few hundred used bytes stay L1-resident).
// The scalars of a parameter record, read as words by one warp.
struct ParamHead {
  float temperature;
  int perim_on;         // any lam_perim != 0
  unsigned fixed_mask;  // bit t: cells of type t never move (src/kernels2d.cu:280-290)
  int stick_on;         // any stickiness != 0
  int chemo_on;         // any chemo != 0
  int act_on;           // any act_lambda != 0
  int persist_on;       // any persist_lambda != 0
  int small_targets;    // all target areas and perimeters within (-2^21, 2^21)
};

struct DevParams : ParamHead {
  float J[kMaxTypes * kMaxTypes];      // J[own type][neighbour type]
  // stickiness S[own type][neighbour type]: added to the adhesion of the
  // configuration before the copy only (src/kernels2d.cu:399-400)
  float stick[kMaxTypes * kMaxTypes];
  float lam_area[kMaxTypes];
  int tgt_area[kMaxTypes];
  float lam_perim[kMaxTypes];
  int tgt_perim[kMaxTypes];
  // chemotaxis lambda per type: dH -= lambda (d . field at the source), d the
  // unit copy direction (src/kernels2d.cu:302-334, src/kernels3d.cu:275-324)
  float chemo[kMaxTypes];
  // act model (src/kernels2d.cu:312-473): lambda and max_act per type;
  // persistence (3D, src/kernels3d.cu:327-343, src/kernels.cu:159-212):
  // lambda and diffusion per type
  float act_lambda[kMaxTypes];
  int act_max[kMaxTypes];
  float persist_lambda[kMaxTypes];
  float persist_diff[kMaxTypes];
  int persist_time[kMaxTypes];  // stored for get/set only (not read by any kernel)
};

// Division of a 31-bit number by a side: n / d = mulhi(n, mul) >> shift, with
// 2^l >= d, mul = floor(2^(31 + l) / d) + 1 and shift = l - 1 (Granlund and
// Montgomery, PLDI'94).
struct FastDiv {
  uint32_t mul, shift;
};
inline FastDiv fast_div_of(uint32_t d) {  // 2 <= d < 2^31
  uint32_t l = 1;
  while ((1ull << l) < d) ++l;
  return {(uint32_t)((1ull << (31 + l)) / d + 1), l - 1};
}

// Quotient and remainder of n < 2^31 by a number of tasks d: with
// inv = floor((2^32 - 1) / d), n * inv / 2^32 lies in (n / d - 1/2, n / d], so the
// product's high word is the quotient or one less.  (Two divisions per task
// were part of what made tasks of 4 rows no better than ones of 8: 4096^2, 50
// MCS 7.09 -> 7.05 ms.)  d is 0 for a replica with no columns of targets in a
// slot that others of its batch have; nothing is divided by it then.
__host__ __device__ inline uint32_t task_reciprocal(int d) {
  return 0xFFFFFFFFu / (uint32_t)(d > 1 ? d : 1);
}
__host__ __device__ inline uint32_t task_quotient(uint32_t n, uint32_t d, uint32_t inv,
                                                  uint32_t& rem) {
#ifdef __CUDA_ARCH__
  uint32_t q = __umulhi(n, inv);
#else
  uint32_t q = (uint32_t)(((uint64_t)n * inv) >> 32);
#endif
  rem = n - q * d;
  if (rem >= d) {
    rem -= d;
    ++q;
  }
  return q;
}

struct DevReplica {
  int nx, ny, nz, ncells;
  long long lat_off;   // first site of the replica in lat[]
  long long cell_off;  // table row of the replica's id 0
  int pset;            // its parameter record in params[] (shared by replicas)
  int pad;
  FastDiv div_nx, div_plane;  // by nx and nx * ny
};

// (area, perimeter) packed in one 64-bit word: area in the low 32 bits (it
// never goes below zero), perimeter in the high 32 bits.  A signed 64-bit
// addition of pack_delta(da, dp) updates both fields exactly.
__host__ __device__ inline unsigned long long pack_delta(int da, int dp) {
  return (unsigned long long)((long long)dp * 4294967296LL + (long long)da);
}
__host__ __device__ inline int unpack_area(unsigned long long w) {
  return (int)(uint32_t)w;
}
__host__ __device__ inline int unpack_perim(unsigned long long w) {
  return (int)(uint32_t)(w >> 32);
}

// Likelihood-ratio scores: up to kScoreMax parameters per replica and MCS,
// in the order (J pairs..., lambda_area, lambda_perim, T).  J pair k is the
// symmetric adhesion of types (pair_a[k], pair_b[k]); only types <
// kScoreTypes enter the derivative.  lambda_area (lambda_perim) is one value
// shared by every cell type's area (perimeter) lambda, each type keeping its
// own target.
constexpr int kScoreMax = 8;
constexpr int kScorePairsMax = 6;
constexpr int kScoreRegs = kScorePairsMax + 3;  // pairs, lambda_area, lambda_perim, T
constexpr int kScoreTypes = 4;
constexpr int kMaxCheckpoints = 64;  // observation times of one backward
struct ScoreSpec {
  int n_pairs;
  int pair_a[kScorePairsMax];
  int pair_b[kScorePairsMax];
  int lambda_area;   // 1: include d/d lambda_area
  int lambda_perim;  // 1: include d/d lambda_perim
  int temperature;   // 1: include d/dT
};

// Arguments of the persistent sweep kernel.
struct SweepArgs {
  uint32_t* lat;
  unsigned long long* ap[2];
  long long* cs[2];
  unsigned long long* dap[2];
  long long* dcs[2];
  uint32_t* dlist;
  uint32_t* ctl;
  unsigned long long* counters;  // [nrep][2]: evaluated, accepted
  const DevReplica* reps;
  const DevParams* params;
  const int* task_prefix;  // (batches) [27][nrep + 1] warp tasks per slot, prefix
  int rows, kr;            // target rows of a task, rows drawn side by side
  long long list_cap;      // entries of one dirty list of one block
  int scan;                // 1: no dirty lists, every table row is replayed
  unsigned scan_rows;      // (batches) rows of the tables
  // Dispatch: 0 = the tiles of every slot over all replicas go to all warps
  // of the grid, one grid barrier per phase; 1 = each block claims whole
  // replicas in rep_order and runs all their phases with block barriers.
  int block_local;
  const int* rep_order;  // replicas by decreasing site count (replica dispatch:
                         // the queue, queue_len entries)
  int queue_len;         // replica dispatch: replicas to claim
  // Grid dispatch over a subset of the replicas (hybrid runs): task_prefix
  // and nrep describe the subset, and rep_map[i] is subset member i's
  // replica (null: the subset is every replica, in order).
  const int* rep_map;
  // chemotaxis field, float: replica r's component k of site i at
  // field[ndim * lat_off + k * sites_r + i] (null when no field exists)
  const float* field;
  // Act model: act[i] = the MCS of the last copy into site i.  With act_on
  // (some record has an act lambda) an attempt also reads around its source,
  // other targets of the slot among it, and must see the phase's starting
  // state.  Lattice and stamps are then double-buffered like the tables: a
  // phase reads one copy, writes its copies into the other and lists them in
  // `pend` (two lists per block: site low, site high, value, stamp); the next
  // phase replays them into the copy they missed.  Both copies are equal
  // before and after a launch.
  // In replica dispatch, whose barriers are a block's, and where the second
  // copies do not fit in memory (16 bytes a site of copies and lists in 2D,
  // against 3) lat2 is null: the blocks list their copies in `pend` (64-bit sites
  // of all blocks, then 32-bit values) and make them after the phase, behind a
  // second barrier.  Two copies / one in grid dispatch (us): 20 MCS of 64^2 598 /
  // 668, of 1024^2 1175 / 1249, of 64^3 785 / 856; one MCS of 4096^2, where
  // starting with equal copies is more of it, 806 / 742.
  uint32_t* act;
  uint32_t* lat2;
  uint32_t* act2;
  int act_on;
  // (3D persistence) preferred direction of each table row, [rows][3]
  const double* prefdir;
  uint4* pend;
  long long pend_cap;  // entries of one pending list of one block
  // Monte Carlo time of the first MCS: tick0, or *tick_ptr when tick_ptr is
  // set (graph replays); in the latter case block 0 advances *tick_ptr by
  // mcs when the launch ends.
  unsigned long long* tick_ptr;
  int tick_advance;  // 0: leave *tick_ptr to a later launch of the same run
  unsigned long long tick0;
  // Score output (score launches only): scores[(r * score_len + tick -
  // score_base) * kScoreMax + k] receives replica r's summed score of
  // parameter k over the attempts of MCS `tick`.
  float* scores;
  unsigned long long score_base;
  int score_len;
  ScoreSpec score_spec;
  unsigned long long seed;
  int nrep;
  int mcs;
  unsigned int stream0;
  int nslot_active;
  int slots[27];
};

// Message returned by cpm_last_error(NULL) for calls without a handle.
void set_thread_error(const char* message);

// Launchers.  Each returns the cudaError_t of its launch.
//
// The sweep (cpm_sweep2d.cu, cpm_sweep3d.cu): batch = grid dispatch over the
// replicas of a batch (a.task_prefix), else one lattice or, with
// a.block_local, whole replicas per block.  At most `warps` warps per block.
cudaError_t launch_sweep2d(const SweepArgs& a, bool batch, bool scores, int grid, int warps,
                           cudaStream_t s);
cudaError_t launch_sweep3d(const SweepArgs& a, bool batch, int grid, int warps, cudaStream_t s);
// Cluster sweep of a small single 2D lattice (cpm_cluster.cu): blocks of the
// cluster that can hold it with its tables (0: none), and launch.  dealt: the
// tables' rows are dealt over the blocks instead of kept by each.
int cluster_sweep_blocks(int nx, int ny, int ncells, bool dealt);
int cluster_sweep_threads();
cudaError_t launch_cluster_sweep(const SweepArgs& a, int nx, int ny, int ncells, int G,
                                 bool dealt, cudaStream_t s);
// checkpoints: host array of ncheck (<= kMaxCheckpoints) MCS counts.
cudaError_t launch_lr_backward(const float* scores, const float* dl_do,
                               const float* obs, const int* checkpoints, int nrep,
                               int len, int nparam, int ncheck, const float* obs_total,
                               int nrep_total, float* grad, cudaStream_t s);
// 3D persistence: initial preferred directions, history fill (push), and
// the update after a run (slot: the history slot that receives this run).
cudaError_t launch_init_prefdir(double* prefdir, const DevReplica* reps, int nrep,
                                long long rows, unsigned long long seed, unsigned stream0,
                                cudaStream_t s);
cudaError_t launch_persist_fill(double* hist, int H, const unsigned long long* ap,
                                const long long* cs, const DevReplica* reps, int nrep,
                                long long rows, cudaStream_t s);
cudaError_t launch_persist_update(double* prefdir, double* hist, int H, int slot,
                                  const unsigned long long* ap, const long long* cs,
                                  const int* ctype, const DevParams* params,
                                  const DevReplica* reps, int nrep, long long rows,
                                  cudaStream_t s);
// Pair counts of 2D replicas; start: per replica its first task of 32 columns
// by kObserveRows rows (nrep + 1 entries, device memory), ntasks = start[nrep].
constexpr int kObserveRows = 16;
cudaError_t launch_observe_heterotypic(const uint32_t* lat, const DevReplica* reps,
                                       int nrep, const long long* start, long long ntasks,
                                       unsigned long long* counts, cudaStream_t s);
// Periodic Voronoi seeding of one lattice region (nx*ny*nz sites at `lat`):
// every site takes values[k] of its nearest point (min-image Euclidean
// distance in double, ties to the lowest k).  Points are binned in a
// g[0]*g[1]*g[2] bucket grid (bucket-major order: pts[k*3+a],
// idx[k] their original index, start[b]..start[b+1] bucket b's points; fpts[k]
// the same coordinates in FP32).
struct VoronoiGrid {
  int n[3];         // lattice sides (n[2] = 1 in 2D)
  int g[3];         // buckets per axis
  double inv[3];    // buckets per unit length, g / n
  double wmin, wmax;  // of the bucket widths n / g: ring r bounds unscanned points at r * wmin
  float inv_w[3];   // the same in FP32
  float wf[3];      // bucket widths in FP32
  float lb_scale;   // wmin in FP32
  float ferr;       // bound on the error of a distance (and of a position) in FP32
  int ndim;
  int rmax;         // rings to scan at most (covers every bucket)
  bool single;      // the rings are scanned in FP32 first
};
// Bucket grid with about two points per bucket.
//
// single: a scan in FP32 goes on until its lower bound, 3 ferr below the true
// one, passes the nearest point, 3 ferr / wmin rings longer than one in double;
// and every point within 2 ferr of the nearest is looked at again.  ferr grows
// with the longest side (0.006 at 4096, 384 at 2^28), wmin with neither.  Up to
// one ring more FP32 is the faster (ms of a call, double / FP32: 256^3 sites,
// 30,000 points 72.8 / 2.7; 2^20 x 8 sites, 80,000 points, half a ring more
// 23.4 / 6.8).  2^28 x 4 sites of 10^7 points would take 288 rings for 7, some
// 6 x 10^14 distances, where the bound on a call's work counts 5 x 10^11: all
// in double there.
inline VoronoiGrid voronoi_grid(int ndim, const int (&n)[3], int npoints) {
  VoronoiGrid vg;
  vg.ndim = ndim;
  const double sites = (double)n[0] * n[1] * n[2];
  const double side = std::pow(2.0 * sites / npoints, 1.0 / ndim);
  vg.wmin = 1e300, vg.wmax = 0.0;
  vg.rmax = 0;
  int nmax = 1;
  for (int a = 0; a < 3; ++a) {
    vg.n[a] = n[a];
    int g = a < ndim ? (int)std::lround((double)n[a] / side) : 1;
    g = std::max(1, std::min(g, n[a]));
    vg.g[a] = g;
    const double w = (double)n[a] / g;
    vg.inv[a] = (double)g / n[a];
    vg.wf[a] = (float)w;
    vg.inv_w[a] = (float)(1.0 / w);
    if (a < ndim) {
      vg.wmin = std::min(vg.wmin, w);
      vg.wmax = std::max(vg.wmax, w);
      nmax = std::max(nmax, n[a]);
    }
    vg.rmax = std::max(vg.rmax, g / 2 + 1);
  }
  vg.lb_scale = (float)vg.wmin;
  // Coordinates and differences of up to nmax, each rounded to FP32 (relative
  // 2^-24): at most 8 roundings per axis, up to sqrt(3) of it in a distance,
  // and a few more of the squares and the square root.
  vg.ferr = (float)(24.0 * nmax * 0x1p-24);
  vg.single = 3.0 * vg.ferr <= vg.wmin;
  return vg;
}
// raw: the points as given; idx: their order by bucket; pts, fpts: room for
// them in that order (filled here); start: first place of each bucket.
cudaError_t launch_voronoi(uint32_t* lat, const VoronoiGrid& vg, int npoints, const double* raw,
                           double* pts, float4* fpts, const int* idx, const uint32_t* values,
                           const int* start, cudaStream_t s);
// Boundary counts per replica and unordered type pair: Moore pairs (each
// once) of sites with different values, counts[r*T*T + a*T + b] for a <= b
// (types >= T are skipped).  tile_start: per replica the first of its tiles
// of kBoundaryTile sites (nrep+1 entries).
constexpr int kBoundaryTile = 4096;
cudaError_t launch_observe_boundaries(int ndim, const uint32_t* lat, const DevReplica* reps,
                                      int nrep, const long long* tile_start,
                                      long long ntiles, int T, unsigned long long* counts,
                                      cudaStream_t s);
cudaError_t launch_barrier_probe(uint32_t* ctl, unsigned long long timeout_ns,
                                 cudaStream_t s);
cudaError_t launch_init(int ndim, const uint32_t* lat, const DevReplica* reps,
                        int nrep, long long total_sites, unsigned long long* ap,
                        long long* cs, unsigned long long* first, int* ctype,
                        uint32_t* ctl, cudaStream_t s);

}  // namespace gpucpm
