// cpm_engine.cu — host runtime of the GB300 Cellular Potts engine and the
// C-ABI of include/gpucpm.h.
//
// Replaces the reference's host class Cpm (src/cpm.h:78-151, src/cpm.cu):
// allocation (src/cpm.cu:176-261), parameter setters (:57-158), addCell
// (:160-174), the launch schedule of run() (:291-517), host<->device copies
// (:531-597) and centroid readback (:68-110).  Differences by design:
//   * one CUDA stream per handle instead of the legacy default stream;
//   * one cooperative persistent launch per run() covers every MCS, slot and
//     replica (the reference relaunches per inner_iterations and grid-syncs
//     per attempt); hybrid-dispatch batches make two;
//   * parameters live in device records shared by replicas (copy on write)
//     and uploaded once per run when changed (the reference re-uploads its
//     __constant__ struct in every setter, src/kernels.cu:50-53);
//   * every call returns a status and keeps a message (the reference prints
//     CUDA errors and carries on, src/cpm.cu:52-56).
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <memory>
#include <string>
#include <vector>

#include "../../include/gpucpm.h"
#include "cpm_internal.h"

using namespace gpucpm;

namespace {

thread_local std::string g_create_error;

constexpr int kMaxMcsPerLaunch = 1 << 16;

}  // namespace

void gpucpm::set_thread_error(const char* message) { g_create_error = message; }

namespace {
constexpr int kWarps2d = 24, kWarpsWide = 20;  // sweep_warps (cpm_sweep.cuh)
}

// Variant 0.  A slot's 32-column rows of targets are spread over every SM.
// While a block has at most one row per warp, one row per task: the phase is
// one warp's chain, and rows side by side would lengthen it.  Up to three rows
// per warp they are drawn side by side, one task per warp, its draws made
// before the phase starts.  Beyond that, 4-row tasks (8-row ones where every
// warp still gets two or more), claimed until the slot is done.  Measured (us,
// 20 MCS, two / three rows side by side): 800^2 518 / 510; 100^3 1143 / 1123;
// 1100 x 1000 634 / 584; 128^3 1354 / 1256; (three / four) 1024^2 956 / 1003;
// (one / two / four) 101 x 75 x 61 box, 20 MCS 2823 / 2827 / 2941;
// 4096^2 tissue, 50 MCS 8755 / 7875 / 7606; 256^3 tissue, 20 MCS 4268 / 3782 /
// 3658 (8-row tasks: 3614).
SweepPlan gpucpm::plan_sweep(int ndim, int nx, int ny, int nz, int variant, int sms, bool wide) {
  const long long ncx = std::max(1, nx >> 1), ncy = std::max(1, ny >> 1),
                  ncz = ndim == 3 ? std::max(1, nz >> 1) : 1;
  const long long tnx = (ncx + 31) / 32, units = tnx * ncy * ncz;
  const int W = ndim == 2 && !wide ? kWarps2d : kWarpsWide;
  const long long upb = (units + sms - 1) / sms;  // rows of a block
  SweepPlan p;
  switch (variant) {
    case 1: p.kr = 4, p.rows = 8; break;
    case 2: p.kr = 4, p.rows = units >= 16LL * sms ? 16 : 8; break;  // (a task per block)
    case 3: p.kr = 1, p.rows = 1; break;
    default:
      p.kr = upb <= W ? 1 : (upb <= 3 * W ? 3 : 4);
      p.rows = upb > 16 * W ? 8 : p.kr;
  }
  if (wide) {
    p.kr = 2;
    p.rows = variant == 0 && upb <= 2 * W ? 2 : std::max(p.rows, 2);
  }
  const long long tasks = tnx * ((ncy + p.rows - 1) / p.rows) * ncz;
  p.grid = (int)std::min<long long>(sms, tasks);
  const long long per = (tasks + p.grid - 1) / p.grid;  // of a block
  p.warps = (int)std::min<long long>(W, per);
  p.list_cap = 2 * std::min(32LL, ncx) * std::min<long long>(p.rows, ncy) * per;
  return p;
}

// Long tasks fill a warp's batches (attempts of different replicas are not
// evaluated together: with queues of two replicas' attempts 256 ragged
// replicas took 3 % longer, their constants no longer being the warp's); small
// batches need every warp to get a task.  Measured (ms): 128 x 256^2 with
// scores 8 rows 24.1, 4 rows 28.1, 16 rows 28.0; 256 ragged replicas 16 rows
// 16.4, 8 rows 19.0; 64 x 64^2 2 rows 0.52, 4 rows 0.59.  The 32 rows of variant 2
// likewise only where every warp gets a task of them (two small 3D replicas, 8
// MCS: 32 rows 3.98 ms, 16 2.67, 8 2.04).
int gpucpm::batch_rows(int variant, long long total_units, int sms) {
  const long long per_warp = total_units / ((long long)sms * kWarpsWide);
  switch (variant) {
    case 1: return 8;
    case 2: return per_warp >= 32 ? 32 : (per_warp >= 1 ? 16 : 8);
    case 3: return 2;
    default: break;
  }
  return per_warp >= 32 ? 16 : (per_warp >= 8 ? 8 : (per_warp >= 4 ? 4 : 2));
}

struct cpm_handle {
  int ndim = 2;
  int nrep = 0;
  int device = 0;
  std::vector<DevReplica> reps;
  // Parameter records shared by replicas (reps[r].pset), copied on the first
  // write that addresses one replica only; records no replica uses are
  // dropped at upload.  A batch whose replicas share their parameters
  // uploads one record.
  std::vector<DevParams> psets;
  std::vector<int> pset_refs;  // replicas using each record
  bool params_dirty = true;
  bool reps_dirty = false;  // some reps[r].pset changed since the last upload
  int params_cap = 0;       // records d_params holds
  long long total_sites = 0;
  long long rows = 0;

  uint32_t* h_lat = nullptr;  // pinned, all replicas back to back
  // chemotaxis field (allocated on first use): host doubles as the
  // reference keeps them, device floats; layout of SweepArgs::field
  std::vector<double> h_field;
  float* d_field = nullptr;
  // act model (allocated on first use): MCS of the last copy into each site;
  // (on the first act run) second copies of lattice and stamps, where they fit,
  // and the blocks' lists of a phase's copies (SweepArgs::lat2, act2, pend)
  std::vector<uint32_t> h_act;
  uint32_t* d_act = nullptr;
  uint32_t* d_lat2 = nullptr;
  uint32_t* d_act2 = nullptr;
  uint4* d_pend = nullptr;
  long long pend_entries = 0;  // of all blocks' lists
  bool act_active = false;     // some replica's record has an act lambda
  // 3D persistence (allocated on first use): preferred direction per table
  // row, and the ring of the cells' mean coordinates after the last runs
  double* d_prefdir = nullptr;  // [rows][3]
  double* d_hist = nullptr;     // [hist_size][rows][3]
  int hist_size = 1;            // the reference's `history` (Cpm constructor)
  int hist_slot = 0;            // slot the next run's means go to
  bool persist_active = false;  // 3D and some record has a persistence lambda
  uint32_t* d_lat = nullptr;
  unsigned long long* d_ap[2] = {nullptr, nullptr};  // packed (area, perimeter)
  long long* d_cs[2] = {nullptr, nullptr};
  unsigned long long* d_dap[2] = {nullptr, nullptr};
  long long* d_dcs[2] = {nullptr, nullptr};
  uint32_t* d_dlist = nullptr;
  uint32_t* d_ctl = nullptr;
  unsigned long long* d_counters = nullptr;
  unsigned long long* d_first = nullptr;
  int* d_ctype = nullptr;
  DevReplica* d_reps = nullptr;
  DevParams* d_params = nullptr;
  int* d_task_prefix = nullptr;
  int* d_hyb_prefix = nullptr;  // [variant][27][nrep + 1] (hybrid grid part)
  int* d_rep_order = nullptr;  // replicas by decreasing site count

  cudaStream_t stream = nullptr;      // stream work is enqueued on
  cudaStream_t own_stream = nullptr;  // created with the handle
  // One launch configuration per tile variant; `variant` is the one runs use
  // (0 until cpm_autotune picks another).  For one lattice `plan` is its
  // sweep's and `wide` that of its extended and score kernels; for a batch
  // both are grid dispatch's, and `local` is replica dispatch's.
  struct Config {
    SweepPlan plan, wide, local;
    std::vector<int> task_prefix;  // (batches) [27][nrep + 1] warp tasks per slot
    std::vector<int> active_slots;
    // hybrid dispatch: the first hyb_ng replicas of rep_order run in grid
    // dispatch (hyb_prefix: [27][hyb_ng + 1], in rep_order), the rest in
    // replica dispatch, a whole number of rounds
    int hyb_ng = 0;
    std::vector<int> hyb_prefix;
  } cfg[kTileVariants];
  int variant = 0;
  bool variant_ext = false;  // the autotuner's choice for act or persistence runs
  int dispatch = CPM_DISPATCH_GRID;  // CPM_DISPATCH_*
  // CPM_FILL_*, as cpm_get_fill tells it.  Until the caller or the autotuner
  // chooses one (fill_by) the engine runs the cluster sweep (cpm_cluster.cu) on
  // small lattices that fit it, else the grid sweep (cpm_sweep.cuh);
  // CPM_FILL_CLUSTER asks for the cluster sweep, the other fills for the grid
  // sweep.  row_ok: the shapes that accept CPM_FILL_VECTOR and CPM_FILL_TMA;
  // cluster_shape: those that accept CPM_FILL_CLUSTER even where their tables
  // do not fit (cluster_blocks = 0) and the grid sweep runs.
  int fill = CPM_FILL_PARITY;
  enum { kBySize, kByTuner, kByCaller } fill_by = kBySize;
  bool row_ok = false, cluster_shape = false;
  int cluster_blocks = 0;  // blocks of the cluster that holds the lattice (0: none)
  bool cluster_dealt = false;  // with the tables' rows dealt over them
  std::vector<unsigned long long> attempts;  // per replica, host-counted

  // Graph-captured run (cpm_run_graph): the captured launch reads and
  // advances the device copy of the tick.
  unsigned long long* d_tick = nullptr;
  bool d_tick_stale = true;
  cudaGraphExec_t graph_exec = nullptr;
  int graph_mcs = 0, graph_variant = -1, graph_dispatch = -1, graph_fill = -1;
  int graph_launches = 1;  // sweep kernels per replay (2 for hybrid)
  cudaStream_t graph_stream = nullptr;

  // Scratch of the synchronous seeding and measuring calls, grown on demand
  // and freed with the handle (an allocation per call costs more than their
  // kernels on small lattices), or at once where it is large (kScratchKept).
  char* d_scratch = nullptr;
  size_t scratch_cap = 0;

  uint64_t seed = 0;
  uint32_t stream_id = 0;
  uint64_t tick = 0;
  bool pushed = false;
  int added_cells = 0;
  uint64_t launches = 0;
  std::string err;

  int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    err = buf;
    return code;
  }
  int cuda_fail(cudaError_t e, const char* what) {
    return fail(CPM_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  }
};

namespace {

#define CPM_CUDA(h, call)                                   \
  do {                                                      \
    cudaError_t e_ = (call);                                \
    if (e_ != cudaSuccess) return (h)->cuda_fail(e_, #call); \
  } while (0)

// Entry points that touch the GPU make the handle's device current first:
// the library carries its own CUDA runtime, whose current device is not the
// one a caller (torch, another library) selected.  What an earlier call of this
// thread failed with (an allocation refused to another engine, say) was
// reported then and is forgotten: the launchers return cudaGetLastError().
#define CPM_BIND(h)                                   \
  do {                                                \
    if (!(h)) return CPM_ERR_INVALID;                 \
    cudaGetLastError();                               \
    CPM_CUDA((h), cudaSetDevice((h)->device));        \
  } while (0)

int class_count_h(int n, int c) {
  if (n == 1) return c == 0 ? 1 : 0;
  return c < 2 ? (n >> 1) : (n & 1);
}

void free_all(cpm_handle* h) {
  if (h->stream) cudaStreamSynchronize(h->stream);
  cudaFreeHost(h->h_lat);
  cudaFree(h->d_field);
  cudaFree(h->d_act);
  cudaFree(h->d_lat2);
  cudaFree(h->d_act2);
  cudaFree(h->d_pend);
  cudaFree(h->d_prefdir);
  cudaFree(h->d_hist);
  cudaFree(h->d_lat);
  for (int b = 0; b < 2; ++b) {
    cudaFree(h->d_ap[b]);
    cudaFree(h->d_cs[b]);
    cudaFree(h->d_dap[b]);
    cudaFree(h->d_dcs[b]);
  }
  cudaFree(h->d_dlist);
  cudaFree(h->d_ctl);
  cudaFree(h->d_counters);
  cudaFree(h->d_first);
  cudaFree(h->d_ctype);
  cudaFree(h->d_reps);
  cudaFree(h->d_params);
  cudaFree(h->d_task_prefix);
  cudaFree(h->d_hyb_prefix);
  cudaFree(h->d_rep_order);
  cudaFree(h->d_tick);
  cudaFree(h->d_scratch);
  if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
  if (h->own_stream) cudaStreamDestroy(h->own_stream);
}

// Shapes that accept CPM_FILL_VECTOR and CPM_FILL_TMA.
bool rows_fit(int ndim, int nx, int ny, int nz) {
  return nx % 4 == 0 && nx >= 72 && (ndim == 2 ? ny >= 66 : ny >= 18 && nz >= 18);
}
// Shapes whose rows alone fit a cluster, about 190 KB of them per block of 16
// (cpm_handle::cluster_shape).
bool cluster_rows_fit(int nx, int ny) {
  if (!rows_fit(2, nx, ny, 1)) return false;
  for (int g : {16, 8}) {
    const long long h = (ny + g - 1) / g;
    const long long strip = (((h + 2) * (nx + 8) + 31) & ~31LL) * 4;
    const long long lists = 8 * (64LL * (((nx >> 1) + 31) / 32) * (h / 2 + 8));
    if (strip + lists + 23040 <= kSweepSmemMax - 1024) return true;
  }
  return false;
}

void default_params(DevParams& p, float T) {
  std::memset(&p, 0, sizeof p);
  p.temperature = T;
}

// Whether every target lies where the sweep may compute a constraint's
// integers in FP32 (DevParams::small_targets).
bool targets_small(const DevParams& p) {
  constexpr int kLim = 1 << 21;
  for (int k = 0; k < kMaxTypes; ++k)
    if (p.tgt_area[k] <= -kLim || p.tgt_area[k] >= kLim || p.tgt_perim[k] <= -kLim ||
        p.tgt_perim[k] >= kLim)
      return false;
  return true;
}

bool perim_on(const DevParams& p) {
  for (int k = 0; k < kMaxTypes; ++k)
    if (p.lam_perim[k] != 0.0f) return true;
  return false;
}

int build_engine(int n, int ndim, const int* nx, const int* ny, const int* nz,
                 const int* ncells, float T, cpm_handle** out) {
  if (!out) {
    g_create_error = "out pointer is NULL";
    return CPM_ERR_INVALID;
  }
  *out = nullptr;
  if (n < 1 || (ndim != 2 && ndim != 3)) {
    g_create_error = "need n >= 1 replicas and dimensionality 2 or 3";
    return CPM_ERR_INVALID;
  }
  cpm_handle* h = new (std::nothrow) cpm_handle();
  if (!h) {
    g_create_error = "host allocation failed";
    return CPM_ERR_ALLOC;
  }
  h->ndim = ndim;
  h->nrep = n;
  long long sites = 0, rows = 0;
  for (int r = 0; r < n; ++r) {
    DevReplica R;
    R.nx = nx[r];
    R.ny = ny[r];
    R.nz = ndim == 3 ? nz[r] : 1;
    R.ncells = ncells[r];
    if (R.nx < 3 || R.ny < 3 || (ndim == 3 && R.nz < 3)) {
      g_create_error = "every side must be at least 3";
      delete h;
      return CPM_ERR_INVALID;
    }
    if (ndim == 2 && nz && nz[r] != 1) {
      g_create_error = "nz must be 1 for a 2D lattice";
      delete h;
      return CPM_ERR_INVALID;
    }
    const long long ns = (long long)R.nx * R.ny * R.nz;
    if (ns >= (1LL << 31)) {
      g_create_error = "a replica may hold at most 2^31-1 sites";
      delete h;
      return CPM_ERR_INVALID;
    }
    if (R.ncells < 0 || R.ncells > 0xFFFFFF) {
      g_create_error = "number_of_cells must be in [0, 2^24-1]";
      delete h;
      return CPM_ERR_INVALID;
    }
    R.lat_off = sites;
    R.cell_off = rows;
    R.pad = 0;
    R.div_nx = fast_div_of((uint32_t)R.nx);
    R.div_plane = fast_div_of((uint32_t)R.nx * (uint32_t)R.ny);
    sites += ns;
    rows += (long long)R.ncells + 1;
    h->reps.push_back(R);
  }
  if (rows >= (1LL << 31)) {
    g_create_error = "too many cells in total (table rows >= 2^31)";
    delete h;
    return CPM_ERR_INVALID;
  }
  h->total_sites = sites;
  h->rows = rows;
  h->psets.resize(1);
  default_params(h->psets[0], T);
  h->pset_refs.assign(1, n);
  for (auto& R : h->reps) R.pset = 0;
  h->attempts.assign(n, 0);

  cudaError_t e = cudaGetDevice(&h->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking);
  h->stream = h->own_stream;
  auto al = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc(p, bytes ? bytes : 1);
  };
  al((void**)&h->d_lat, sizeof(uint32_t) * sites);
  for (int b = 0; b < 2; ++b) {
    al((void**)&h->d_ap[b], sizeof(unsigned long long) * rows);
    al((void**)&h->d_cs[b], sizeof(long long) * rows * ndim);
    al((void**)&h->d_dap[b], sizeof(unsigned long long) * rows);
    al((void**)&h->d_dcs[b], sizeof(long long) * rows * ndim);
  }
  al((void**)&h->d_ctl, sizeof(uint32_t) * kCtlWords);
  al((void**)&h->d_counters, sizeof(unsigned long long) * 2 * n);
  al((void**)&h->d_first, sizeof(unsigned long long) * rows);
  al((void**)&h->d_ctype, sizeof(int) * rows);
  al((void**)&h->d_reps, sizeof(DevReplica) * n);
  al((void**)&h->d_params, sizeof(DevParams));
  h->params_cap = 1;
  if (n > 1) {
    al((void**)&h->d_task_prefix, sizeof(int) * kTileVariants * 27 * (n + 1));
    al((void**)&h->d_hyb_prefix, sizeof(int) * kTileVariants * 27 * (n + 1));
  }
  al((void**)&h->d_rep_order, sizeof(int) * n);
  al((void**)&h->d_tick, sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMallocHost((void**)&h->h_lat, sizeof(uint32_t) * (sites ? sites : 1));
  if (e != cudaSuccess) {
    g_create_error = std::string("device/pinned allocation failed: ") + cudaGetErrorString(e);
    free_all(h);
    delete h;
    return e == cudaErrorMemoryAllocation ? CPM_ERR_ALLOC : CPM_ERR_CUDA;
  }
  std::memset(h->h_lat, 0, sizeof(uint32_t) * sites);
  if (n == 1 && rows_fit(ndim, nx[0], ny[0], nz ? nz[0] : 1)) {
    h->row_ok = true;
    h->fill = CPM_FILL_TMA;
    if (ndim == 2) h->cluster_shape = cluster_rows_fit(nx[0], ny[0]);
  }
  if (n == 1 && ndim == 2) {
    h->cluster_blocks = cluster_sweep_blocks(nx[0], ny[0], ncells[0], false);
    if (h->cluster_blocks == 0) {
      h->cluster_blocks = cluster_sweep_blocks(nx[0], ny[0], ncells[0], true);
      h->cluster_dealt = h->cluster_blocks > 0;
    }
  }

  // One launch configuration per tile variant: warp tasks per slot and
  // replica (prefix over replicas), grid, dirty-list capacity.
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
  long long dlist_entries = 1;
  long long max_rows = 1, max_sites = 1;
  for (const DevReplica& R : h->reps) {
    max_rows = std::max(max_rows, (long long)R.ncells + 1);
    max_sites = std::max(max_sites, (long long)R.nx * R.ny * R.nz);
  }
  std::vector<int> order(n);
  for (int r = 0; r < n; ++r) order[r] = r;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    const DevReplica &X = h->reps[x], &Y = h->reps[y];
    return (long long)X.nx * X.ny * X.nz > (long long)Y.nx * Y.ny * Y.nz;
  });
  // 32-column rows of targets of replica r's slot
  auto units = [&](int r, int slot, int rows) -> long long {
    const DevReplica& R = h->reps[r];
    const int cx = slot % 3, cy = (slot / 3) % 3, cz = slot / 9;
    if (ndim == 2 && cz != 0) return 0;
    const long long ncx = class_count_h(R.nx, cx), ncy = class_count_h(R.ny, cy),
                    ncz = class_count_h(R.nz, cz);
    return ((ncx + 31) / 32) * ((ncy + rows - 1) / rows) * ncz;
  };
  if (sms < 1) {
    g_create_error = "cannot place the sweep kernel on this device";
    free_all(h);
    delete h;
    return CPM_ERR_CUDA;
  }
  long long total_units = 0;
  int biggest = order[0];
  for (int r = 0; r < n; ++r) {
    total_units += units(r, 0, 1);
    if (units(r, 0, 1) > units(biggest, 0, 1)) biggest = r;
  }
  long long pend_entries = 1;
  for (int v = 0; v < kTileVariants; ++v) {
    cpm_handle::Config& c = h->cfg[v];
    const DevReplica& B = h->reps[biggest];
    if (n == 1) {
      c.plan = plan_sweep(ndim, B.nx, B.ny, B.nz, v, sms, false);
      c.wide = plan_sweep(ndim, B.nx, B.ny, B.nz, v, sms, true);
      c.local = c.plan;  // (not used)
      dlist_entries = std::max(dlist_entries, c.plan.list_cap * 2 * c.plan.grid);
      dlist_entries = std::max(dlist_entries, c.wide.list_cap * 2 * c.wide.grid);
      pend_entries = std::max(pend_entries, c.wide.list_cap * c.wide.grid);
    }
    const int rows = n == 1 ? c.plan.rows : batch_rows(v, total_units, sms);
    if (n > 1) c.task_prefix.assign(27 * (n + 1), 0);
    long long max_tasks = 1;
    for (int slot = 0; slot < 27; ++slot) {
      long long acc = 0;
      for (int r = 0; r < n; ++r) {
        if (n > 1)
          c.task_prefix[slot * (n + 1) + r] = (int)std::min<long long>(acc, INT32_MAX);
        acc += units(r, slot, rows);
      }
      if (acc >= (1LL << 31)) {
        g_create_error = "batch too large for one launch";
        free_all(h);
        delete h;
        return CPM_ERR_INVALID;
      }
      if (n > 1) c.task_prefix[slot * (n + 1) + n] = (int)acc;
      if (acc > 0) c.active_slots.push_back(slot);
      max_tasks = std::max(max_tasks, acc);
    }
    if (n > 1) {
      // Grid dispatch: tasks dealt one at a time, at most ceil(tasks / grid)
      // per block, each attempt touching at most two table rows.
      c.plan.kr = rows >= 4 ? 4 : 2;
      c.plan.rows = rows;
      c.plan.warps = 20;
      c.plan.grid = (int)std::min<long long>(sms, max_tasks);
      c.plan.list_cap = 2LL * 32 * rows * ((max_tasks + c.plan.grid - 1) / c.plan.grid);
      c.wide = c.plan;
      // Replica dispatch: one block per replica at a time.
      // Fixed rows only where every warp gets a task of them (200 replicas of up to
      // 60^2, one MCS in 16-row tasks 178 us, in these 64), one-row tasks only
      // where that is not what the size gives anyway.
      const long long fixed = units(biggest, 0, 1) / kWarps2d;  // rows per warp
      const int lv = fixed < (v == 3 ? 3 : (v == 2 ? 16 : 8)) ? 0 : v;
      c.local = plan_sweep(ndim, B.nx, B.ny, B.nz, lv, 1, false);
      const SweepPlan w = plan_sweep(ndim, B.nx, B.ny, B.nz, lv, 1, true);
      c.local.list_cap = std::max(c.local.list_cap, w.list_cap);
      for (int r = 0; r < n; ++r)  // (a narrower replica may have more rows)
        c.local.list_cap = std::max(c.local.list_cap, 2LL * 32 * c.local.rows *
                                                          units(r, 0, c.local.rows));
      c.local.grid = std::min(sms, n);
      for (const SweepPlan& p : {c.plan, c.local}) {
        dlist_entries = std::max(dlist_entries, p.list_cap * 2 * p.grid);
        pend_entries = std::max(pend_entries, p.list_cap * p.grid);
      }
    }
    if (n == 1) continue;
    // Hybrid split: replica dispatch gets whole rounds of the smallest
    // replicas, grid dispatch the rest.
    c.hyb_ng = n - (n / c.local.grid) * c.local.grid;
    const int ng = c.hyb_ng;
    c.hyb_prefix.assign(27 * (ng + 1), 0);
    for (int slot = 0; slot < 27; ++slot) {
      int acc = 0;
      for (int i = 0; i < ng; ++i) {
        c.hyb_prefix[slot * (ng + 1) + i] = acc;
        const int r = order[i];
        acc += c.task_prefix[slot * (n + 1) + r + 1] - c.task_prefix[slot * (n + 1) + r];
      }
      c.hyb_prefix[slot * (ng + 1) + ng] = acc;
    }
  }
  // act runs list one copy per attempt at most, half of a dirty list's
  // entries, in two lists per block (one where there is one lattice copy)
  h->pend_entries = pend_entries;
  e = cudaMalloc((void**)&h->d_dlist, sizeof(uint32_t) * dlist_entries);
  if (e != cudaSuccess) {
    g_create_error = std::string("dirty-list allocation failed: ") + cudaGetErrorString(e);
    free_all(h);
    delete h;
    return e == cudaErrorMemoryAllocation ? CPM_ERR_ALLOC : CPM_ERR_CUDA;
  }

  // Replica dispatch by default when there are replicas for every block and
  // no replica is much larger than a block's fair share of the sites, hybrid
  // when those replicas do not fill whole rounds (the autotuner can change
  // the choice).
  h->dispatch = (n >= h->cfg[0].local.grid && n >= sms &&
                 max_sites * (long long)h->cfg[0].local.grid <= 2 * sites)
                    ? (h->cfg[0].hyb_ng > 0 ? CPM_DISPATCH_HYBRID : CPM_DISPATCH_REPLICA)
                    : CPM_DISPATCH_GRID;
  e = cudaMemcpyAsync(h->d_reps, h->reps.data(), sizeof(DevReplica) * n,
                      cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h->d_rep_order, order.data(), sizeof(int) * n,
                        cudaMemcpyHostToDevice, h->stream);
  for (int v = 0; n > 1 && v < kTileVariants && e == cudaSuccess; ++v) {
    e = cudaMemcpyAsync(h->d_task_prefix + (size_t)v * 27 * (n + 1),
                        h->cfg[v].task_prefix.data(), sizeof(int) * 27 * (n + 1),
                        cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(h->d_hyb_prefix + (size_t)v * 27 * (n + 1),
                          h->cfg[v].hyb_prefix.data(),
                          sizeof(int) * h->cfg[v].hyb_prefix.size(), cudaMemcpyHostToDevice,
                          h->stream);
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(h->d_ctl, 0, sizeof(uint32_t) * kCtlWords, h->stream);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(h->d_counters, 0, sizeof(unsigned long long) * 2 * n, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) {
    g_create_error = std::string("initial upload failed: ") + cudaGetErrorString(e);
    free_all(h);
    delete h;
    return CPM_ERR_CUDA;
  }
  *out = h;
  return CPM_OK;
}

int check_replica(cpm_handle* h, int r) {
  if (!h) return CPM_ERR_INVALID;
  if (r < 0 || r >= h->nrep)
    return h->fail(CPM_ERR_INVALID, "replica %d out of range [0, %d)", r, h->nrep);
  return CPM_OK;
}

int check_type(cpm_handle* h, int t) {
  if (t < 0 || t >= kMaxTypes)
    return h->fail(CPM_ERR_INVALID, "cell type %d out of range [0, %d)", t, kMaxTypes);
  return CPM_OK;
}

template <class F>
int for_replicas(cpm_handle* h, int r, F&& f) {
  if (!h) return CPM_ERR_INVALID;
  if (r == -1) {
    for (size_t i = 0; i < h->psets.size(); ++i)
      if (h->pset_refs[i] > 0) f(h->psets[i]);
  } else {
    if (int rc = check_replica(h, r)) return rc;
    int p = h->reps[r].pset;
    if (h->pset_refs[p] > 1) {  // shared: give replica r its own copy
      h->psets.push_back(h->psets[p]);
      h->pset_refs.push_back(1);
      --h->pset_refs[p];
      p = (int)h->psets.size() - 1;
      h->reps[r].pset = p;
      h->reps_dirty = true;
    }
    f(h->psets[p]);
  }
  h->params_dirty = true;
  return CPM_OK;
}

int set_temperature(cpm_handle* h, int r, float T) {
  if (!h) return CPM_ERR_INVALID;
  if (!std::isfinite(T)) return h->fail(CPM_ERR_INVALID, "temperature must be finite");
  return for_replicas(h, r, [&](DevParams& p) { p.temperature = T; });
}

int set_area(cpm_handle* h, int r, int type, int target, float lambda) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  return for_replicas(h, r, [&](DevParams& p) {
    p.tgt_area[type] = target;
    p.lam_area[type] = lambda;
  });
}

int set_perimeter(cpm_handle* h, int r, int type, int target, float lambda) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  return for_replicas(h, r, [&](DevParams& p) {
    p.tgt_perim[type] = target;
    p.lam_perim[type] = lambda;
    p.perim_on = perim_on(p) ? 1 : 0;
  });
}

int set_fixed(cpm_handle* h, int r, int type, int fixed) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  return for_replicas(h, r, [&](DevParams& p) {
    if (fixed)
      p.fixed_mask |= 1u << type;
    else
      p.fixed_mask &= ~(1u << type);
  });
}

int set_stickiness(cpm_handle* h, int r, int type, int other, float S) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  if (int rc = check_type(h, other)) return rc;
  if (!std::isfinite(S)) return h->fail(CPM_ERR_INVALID, "stickiness must be finite");
  return for_replicas(h, r, [&](DevParams& p) { p.stick[type * kMaxTypes + other] = S; });
}

int set_adhesion(cpm_handle* h, int r, int type, int other, float J, int sym) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  if (int rc = check_type(h, other)) return rc;
  return for_replicas(h, r, [&](DevParams& p) {
    p.J[type * kMaxTypes + other] = J;
    if (sym) p.J[other * kMaxTypes + type] = J;
  });
}

// At least `bytes` of scratch at h->d_scratch.  Its users wait for the stream
// before they return, so nothing in flight holds the old one, and trim it then.
int ensure_scratch(cpm_handle* h, size_t bytes) {
  if (bytes <= h->scratch_cap) return CPM_OK;
  cudaFree(h->d_scratch);
  h->d_scratch = nullptr;
  h->scratch_cap = 0;
  CPM_CUDA(h, cudaMalloc((void**)&h->d_scratch, bytes));
  h->scratch_cap = bytes;
  return CPM_OK;
}

// Gives back scratch that is large enough to be missed (256 MB: the points of a
// seeding from 4 million, calls in which the allocation does not show: 4096^2
// sites from 4.4 million points 53.7 ms, with the scratch kept 54.7).
constexpr size_t kScratchKept = (size_t)256 << 20;
void trim_scratch(cpm_handle* h) {
  if (h->scratch_cap <= kScratchKept) return;
  cudaFree(h->d_scratch);
  h->d_scratch = nullptr;
  h->scratch_cap = 0;
}

int read_error_word(cpm_handle* h, uint32_t* word) {
  CPM_CUDA(h, cudaMemcpyAsync(word, h->d_ctl + kCtlErr, sizeof(uint32_t),
                              cudaMemcpyDeviceToHost, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  return CPM_OK;
}

// Persistence buffers on first use: directions drawn from (seed, stream),
// history filled from the current tables when they exist.
int ensure_persist(cpm_handle* h) {
  if (!h->d_prefdir) {
    CPM_CUDA(h, cudaMalloc((void**)&h->d_prefdir, sizeof(double) * 3 * h->rows));
    CPM_CUDA(h, launch_init_prefdir(h->d_prefdir, h->d_reps, h->nrep, h->rows, h->seed,
                                    h->stream_id, h->stream));
  }
  if (!h->d_hist) {
    CPM_CUDA(h, cudaMalloc((void**)&h->d_hist, sizeof(double) * 3 * h->rows * h->hist_size));
    CPM_CUDA(h, cudaMemsetAsync(h->d_hist, 0, sizeof(double) * 3 * h->rows * h->hist_size,
                                h->stream));
    h->hist_slot = 0;
    if (h->pushed)
      CPM_CUDA(h, launch_persist_fill(h->d_hist, h->hist_size, h->d_ap[0], h->d_cs[0], h->d_reps,
                                      h->nrep, h->rows, h->stream));
  }
  return CPM_OK;
}

// After a run of a persistence engine: the cells' means into the history,
// and the preferred directions updated (src/cpm.cu:486-510).
int persist_after_run(cpm_handle* h) {
  if (!h->persist_active) return CPM_OK;
  CPM_CUDA(h, launch_persist_update(h->d_prefdir, h->d_hist, h->hist_size, h->hist_slot,
                                    h->d_ap[0], h->d_cs[0], h->d_ctype, h->d_params, h->d_reps,
                                    h->nrep, h->rows, h->stream));
  h->launches += 1;
  h->hist_slot = (h->hist_slot + 1) % h->hist_size;
  return CPM_OK;
}

// The act lattice (zeros), on first use.
int ensure_act(cpm_handle* h) {
  if (!h->d_act) {
    const size_t n = (size_t)h->total_sites;
    try {
      h->h_act.assign(n, 0u);
    } catch (...) {
      return h->fail(CPM_ERR_ALLOC, "host act lattice allocation failed");
    }
    CPM_CUDA(h, cudaMalloc((void**)&h->d_act, sizeof(uint32_t) * (n ? n : 1)));
    CPM_CUDA(h, cudaMemsetAsync(h->d_act, 0, sizeof(uint32_t) * (n ? n : 1), h->stream));
  }
  return CPM_OK;
}

// The act run's second lattice and stamp copies and its lists; where these do
// not fit, the lists of a run with one copy alone.
int ensure_act_run(cpm_handle* h) {
  if (int rc = ensure_act(h)) return rc;
  if (h->d_pend) return CPM_OK;
  const size_t b = sizeof(uint32_t) * (h->total_sites ? h->total_sites : 1);
  cudaError_t e = cudaMalloc((void**)&h->d_lat2, b);
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_act2, b);
  if (e == cudaSuccess) e = cudaMalloc((void**)&h->d_pend, sizeof(uint4) * h->pend_entries);
  if (e == cudaSuccess) return CPM_OK;
  cudaFree(h->d_lat2);
  cudaFree(h->d_act2);
  h->d_lat2 = h->d_act2 = nullptr;
  h->d_pend = nullptr;
  if (e != cudaErrorMemoryAllocation) return h->cuda_fail(e, "allocation of the act run's copies");
  cudaGetLastError();  // (not an error of the run)
  const size_t entries = (size_t)(h->pend_entries + 1) / 2;
  CPM_CUDA(h, cudaMalloc((void**)&h->d_pend,
                         (sizeof(unsigned long long) + sizeof(uint32_t)) * entries));
  return CPM_OK;
}

int upload_params(cpm_handle* h) {
  if (!h->params_dirty && !h->reps_dirty) return CPM_OK;
  // Drop records no replica uses and renumber the rest.
  const int n0 = (int)h->psets.size();
  std::vector<int> remap(n0, -1);
  int m = 0;
  for (int i = 0; i < n0; ++i) {
    if (h->pset_refs[i] <= 0) continue;
    remap[i] = m;
    if (m != i) {
      h->psets[m] = h->psets[i];
      h->pset_refs[m] = h->pset_refs[i];
    }
    ++m;
  }
  if (m != n0) {
    h->psets.resize(m);
    h->pset_refs.resize(m);
    for (auto& R : h->reps) R.pset = remap[R.pset];
    h->reps_dirty = true;
  }
  for (auto& p : h->psets) {
    p.perim_on = perim_on(p) ? 1 : 0;
    p.stick_on = 0;
    for (int k = 0; k < kMaxTypes * kMaxTypes; ++k)
      if (p.stick[k] != 0.0f) p.stick_on = 1;
    p.chemo_on = 0;
    for (int k = 0; k < kMaxTypes; ++k)
      if (p.chemo[k] != 0.0f) p.chemo_on = 1;
    if (p.chemo_on && !h->d_field)
      return h->fail(CPM_ERR_STATE, "chemotaxis is set but the engine has no field "
                                    "(create it with the field flag or call cpm_host_field_r)");
    p.act_on = 0;
    for (int k = 0; k < kMaxTypes; ++k)
      if (p.act_lambda[k] != 0.0f) p.act_on = 1;
    p.persist_on = 0;
    for (int k = 0; k < kMaxTypes; ++k)
      if (p.persist_lambda[k] != 0.0f) p.persist_on = 1;
    p.small_targets = targets_small(p) ? 1 : 0;
  }
  bool persist = false;
  for (const auto& p : h->psets) persist = persist || (h->ndim == 3 && p.persist_on);
  if (persist) {
    if (int rc = ensure_persist(h)) return rc;
  }
  if (persist != h->persist_active) {
    h->persist_active = persist;
    if (h->graph_exec) {
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
  }
  bool act = false;
  for (const auto& p : h->psets) act = act || p.act_on;
  if (act) {
    if (int rc = ensure_act_run(h)) return rc;
  }
  if (act != h->act_active) {  // another kernel, other arguments
    h->act_active = act;
    if (h->graph_exec) {
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
  }
  if (m > h->params_cap) {
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree(h->d_params);
    h->d_params = nullptr;
    h->params_cap = 0;
    CPM_CUDA(h, cudaMalloc((void**)&h->d_params, sizeof(DevParams) * m));
    h->params_cap = m;
    if (h->graph_exec) {  // it holds the old address
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
  }
  CPM_CUDA(h, cudaMemcpyAsync(h->d_params, h->psets.data(), sizeof(DevParams) * m,
                              cudaMemcpyHostToDevice, h->stream));
  if (h->reps_dirty)
    CPM_CUDA(h, cudaMemcpyAsync(h->d_reps, h->reps.data(), sizeof(DevReplica) * h->nrep,
                                cudaMemcpyHostToDevice, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));  // the host copies may change next
  h->params_dirty = false;
  h->reps_dirty = false;
  return CPM_OK;
}

// Whether a sweep looks at every table row instead of keeping dirty lists:
// with up to a row per eight sites the coalesced scan costs less than the
// lists (us per 20 MCS of 1024^2, scan / lists, at a row per 100 sites 547 /
// 544, per 25 726 / 766, per 9 823 / 889, per 5 876 / 912; 100^3 per 9 1852 /
// 1894).  A lattice with more rows than that keeps most of them for cells to
// come, whose rows the lists never see.
bool scans(const cpm_handle* h) { return 8 * h->rows <= h->total_sites; }

// The variant that runs use.  A caller's choice is one for plain runs and
// scores: runs with the act or persistence term take variant 0, or what the
// autotuner timed on such runs (160 small replicas with act, 8 MCS: 0.84 ms, in
// variant 2 3.80).
int run_variant(const cpm_handle* h) {
  return (h->act_active || h->persist_active) && !h->variant_ext ? 0 : h->variant;
}

// Kernel arguments of a sweep with tile variant v and dispatch d (tick0 /
// mcs, and what depends on the launch, filled in by the caller).
SweepArgs sweep_args(const cpm_handle* h, int v) {
  SweepArgs a;
  std::memset(&a, 0, sizeof a);
  a.lat = h->d_lat;
  for (int b = 0; b < 2; ++b) {
    a.ap[b] = h->d_ap[b];
    a.cs[b] = h->d_cs[b];
    a.dap[b] = h->d_dap[b];
    a.dcs[b] = h->d_dcs[b];
  }
  const cpm_handle::Config& c = h->cfg[v];
  a.dlist = h->d_dlist;
  a.scan = scans(h) ? 1 : 0;
  a.scan_rows = (unsigned)h->rows;
  a.field = h->d_field;
  a.act_on = h->act_active ? 1 : 0;
  if (h->act_active) {
    a.act = h->d_act;
    a.lat2 = h->d_lat2;
    a.act2 = h->d_act2;
    a.pend = h->d_pend;
  }
  a.prefdir = h->persist_active ? h->d_prefdir : nullptr;
  a.rep_order = h->d_rep_order;
  a.queue_len = h->nrep;
  a.rep_map = nullptr;
  a.tick_advance = 1;
  a.ctl = h->d_ctl;
  a.counters = h->d_counters;
  a.reps = h->d_reps;
  a.params = h->d_params;
  if (h->nrep > 1) a.task_prefix = h->d_task_prefix + (size_t)v * 27 * (h->nrep + 1);
  a.seed = h->seed;
  a.nrep = h->nrep;
  a.stream0 = h->stream_id;
  a.nslot_active = (int)c.active_slots.size();
  for (int i = 0; i < a.nslot_active; ++i) a.slots[i] = c.active_slots[i];
  return a;
}

// The plan of a launch with variant v and dispatch d (GRID or REPLICA).
const SweepPlan& plan_of(const cpm_handle* h, int v, int d, bool scores = false) {
  const cpm_handle::Config& c = h->cfg[v];
  if (d == CPM_DISPATCH_REPLICA) return c.local;
  return scores || h->act_active || h->persist_active ? c.wide : c.plan;
}

int grid_of(const cpm_handle* h, int v, int d) { return plan_of(h, v, d).grid; }

int fill_key(const cpm_handle* h) { return h->fill_by == cpm_handle::kBySize ? -2 : h->fill; }

// Whether plain runs take the cluster sweep.
// By itself up to about the size where the grid sweep, whose phases take 4.6 us
// whatever the size, overtakes its 16 SMs.  The line is that of the sorting
// lattice (us per MCS, grid / cluster: 350^2 19.5 / 16.7, 400^2 19.2 / 20.4).
// Dense tissues cross it earlier, and long lattices, whose rows or columns do
// not divide evenly over 16 blocks, here and there (tissue of 50 sites a cell:
// 330^2 18.6 / 19.9, 4000 x 16 18.3 / 20.4, 100 x 1300 18.7 / 21.0, but 16 x 4000
// 18.0 / 11.8, 2000 x 32 18.4 / 12.4, 4095 x 5 32.2 / 26.1).
constexpr long long kClusterAutoSites = 140000;
// Where a block cannot hold whole tables they are dealt over the blocks, at a
// second cluster barrier per phase: by the autotuner's choice, or where the
// caller asks for the cluster on lattices so small that it is the faster one
// (us of 20 MCS, grid / dealt, cells of 2 sites and of 25 with 16,000 rows to
// spare: 120 x 173 580 / 371, 532 / 334; 160^2 426 / 310, 396 / 254; 200^2 434 /
// 446, 408 / 310; 256^2 437 / 522, 411 / 421; before, with tables in global memory,
// 200^2 485 and 373).
constexpr long long kClusterDealtSites = 45000;
bool uses_cluster(const cpm_handle* h) {
  if (h->cluster_blocks == 0 || h->act_active || h->persist_active) return false;
  switch (h->fill_by) {
    case cpm_handle::kBySize: return !h->cluster_dealt && h->total_sites <= kClusterAutoSites;
    case cpm_handle::kByTuner: return h->fill == CPM_FILL_CLUSTER;
    default:
      return h->fill == CPM_FILL_CLUSTER &&
             (!h->cluster_dealt || h->total_sites <= kClusterDealtSites);
  }
}

// The launches of one sweep run (`a` from sweep_args, times filled in): one
// launch for GRID and REPLICA, two for HYBRID (grid dispatch over the first
// hyb_ng replicas of rep_order, then replica dispatch over the rest).  Each
// launch starts with its barrier words cleared.  Returns the number of
// launches through *nlaunch.
cudaError_t enqueue_sweep(const cpm_handle* h, int v, int d, const SweepArgs& a, bool scores,
                          int* nlaunch) {
  const cpm_handle::Config& c = h->cfg[v];
  *nlaunch = 0;
  auto one = [&](SweepArgs x, const SweepPlan& p, bool batch) {
    cudaError_t e;
    if (uses_cluster(h) && !scores) {  // (no grid barrier, no queue)
      const DevReplica& R = h->reps[0];
      e = launch_cluster_sweep(x, R.nx, R.ny, R.ncells, h->cluster_blocks, h->cluster_dealt,
                               h->stream);
    } else {
      e = cudaMemsetAsync(h->d_ctl, 0, sizeof(uint32_t) * kCtlErr, h->stream);
      if (x.lat2) {  // both lattice and stamp copies start equal
        const size_t b = sizeof(uint32_t) * h->total_sites;
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(x.lat2, x.lat, b, cudaMemcpyDeviceToDevice, h->stream);
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(x.act2, x.act, b, cudaMemcpyDeviceToDevice, h->stream);
      }
      if (e != cudaSuccess) return e;
      x.rows = p.rows;
      x.kr = p.kr;
      x.list_cap = p.list_cap;
      x.pend_cap = p.list_cap / 2;
      e = h->ndim == 2 ? launch_sweep2d(x, batch, scores, p.grid, p.warps, h->stream)
                       : launch_sweep3d(x, batch, p.grid, p.warps, h->stream);
    }
    if (e == cudaSuccess) ++*nlaunch;
    return e;
  };
  if (d == CPM_DISPATCH_GRID) {
    SweepArgs g = a;
    g.block_local = 0;
    return one(g, plan_of(h, v, d, scores), h->nrep > 1);
  }
  const int ng = d == CPM_DISPATCH_HYBRID ? c.hyb_ng : 0;
  if (ng > 0) {  // grid dispatch over the largest replicas
    SweepArgs g = a;
    g.block_local = 0;
    g.nrep = ng;
    g.task_prefix = h->d_hyb_prefix + (size_t)v * 27 * (h->nrep + 1);
    g.rep_map = h->d_rep_order;
    g.tick_advance = ng < h->nrep ? 0 : 1;
    if (cudaError_t e = one(g, c.plan, true)) return e;
  }
  if (ng < h->nrep) {  // replica dispatch over the rest
    SweepArgs q = a;
    q.block_local = 1;
    // Act: one copy, as the second barrier of a phase is only the block's (us,
    // two copies / one: 40 x 64^2, 10 MCS 363 / 335, 160 x 64^2 621 / 581, and two
    // almost frozen lattices of 1,700 sites, one MCS 68 / 54).
    q.lat2 = q.act2 = nullptr;
    q.rep_order = h->d_rep_order + ng;
    q.queue_len = h->nrep - ng;
    if (cudaError_t e = one(q, c.local, false)) return e;
  }
  return cudaSuccess;
}

void count_attempts(cpm_handle* h, int mcs) {
  for (int r = 0; r < h->nrep; ++r) {
    const DevReplica& R = h->reps[r];
    h->attempts[r] += (unsigned long long)R.nx * R.ny * R.nz * (unsigned long long)mcs;
  }
}

std::string describe_errors(uint32_t w) {
  std::string s;
  auto add = [&](const char* m) {
    if (!s.empty()) s += "; ";
    s += m;
  };
  if (w & kErrBadId) add("a site holds an id above number_of_cells");
  if (w & kErrBadType) add("a site holds a type >= 32");
  if (w & kErrMediumType) add("a site holds id 0 with a non-zero type");
  if (w & kErrTypeConflict) add("one cell id appears with two different types");
  if (w & kErrTimeout) add("a grid barrier of the sweep timed out");
  if (w & kErrListFull) add("a dirty list of the sweep was too small (internal error)");
  return s;
}

}  // namespace

extern "C" {

int cpm_create(int dimension, int dimensionality, int number_of_cells,
               float temperature, int flags, cpm_handle** out) {
  if (flags & ~(CPM_FLAG_FIELD | CPM_FLAG_ACT)) {
    g_create_error = "unknown flags (CPM_FLAG_FIELD and CPM_FLAG_ACT are the flags)";
    if (out) *out = nullptr;
    return CPM_ERR_UNSUPPORTED;
  }
  const int nz = dimensionality == 3 ? dimension : 1;
  const int rc = build_engine(1, dimensionality, &dimension, &dimension, &nz,
                              &number_of_cells, temperature, out);
  if (rc == CPM_OK && (flags & CPM_FLAG_FIELD)) {
    if (int rc2 = cpm_host_field_r(*out, 0, nullptr, nullptr)) {
      g_create_error = cpm_last_error(*out);
      cpm_destroy(*out);
      *out = nullptr;
      return rc2;
    }
  }
  if (rc == CPM_OK && (flags & CPM_FLAG_ACT)) {
    if (int rc2 = cpm_host_act_r(*out, 0, nullptr, nullptr)) {
      g_create_error = cpm_last_error(*out);
      cpm_destroy(*out);
      *out = nullptr;
      return rc2;
    }
  }
  return rc;
}

int cpm_create_box(int nx, int ny, int nz, int dimensionality,
                   int number_of_cells, float temperature, cpm_handle** out) {
  return build_engine(1, dimensionality, &nx, &ny, &nz, &number_of_cells,
                      temperature, out);
}

int cpm_create_batch(int n, int dimensionality, const int* nx, const int* ny,
                     const int* nz, const int* ncells, cpm_handle** out) {
  if (!nx || !ny || !ncells || (dimensionality == 3 && !nz)) {
    g_create_error = "nx, ny, ncells (and nz in 3D) must be non-NULL";
    if (out) *out = nullptr;
    return CPM_ERR_INVALID;
  }
  return build_engine(n, dimensionality, nx, ny, nz, ncells, 1.0f, out);
}

int cpm_destroy(cpm_handle* h) {
  if (!h) return CPM_OK;
  cudaSetDevice(h->device);
  free_all(h);
  delete h;
  return CPM_OK;
}

int cpm_set_device(int device) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) {
    g_create_error = std::string("cudaSetDevice failed: ") + cudaGetErrorString(e);
    return CPM_ERR_CUDA;
  }
  return CPM_OK;
}

const char* cpm_last_error(const cpm_handle* h) {
  return h ? h->err.c_str() : g_create_error.c_str();
}

int cpm_set_temperature(cpm_handle* h, float T) { return set_temperature(h, -1, T); }
int cpm_set_temperature_r(cpm_handle* h, int r, float T) { return set_temperature(h, r < 0 ? -2 : r, T); }
int cpm_set_area(cpm_handle* h, int type, int target, float lambda) {
  return set_area(h, -1, type, target, lambda);
}
int cpm_set_area_r(cpm_handle* h, int r, int type, int target, float lambda) {
  return set_area(h, r < 0 ? -2 : r, type, target, lambda);
}
int cpm_set_perimeter(cpm_handle* h, int type, int target, float lambda) {
  return set_perimeter(h, -1, type, target, lambda);
}
int cpm_set_perimeter_r(cpm_handle* h, int r, int type, int target, float lambda) {
  return set_perimeter(h, r < 0 ? -2 : r, type, target, lambda);
}
int cpm_set_fixed(cpm_handle* h, int type, int fixed) { return set_fixed(h, -1, type, fixed); }
int cpm_set_fixed_r(cpm_handle* h, int r, int type, int fixed) {
  return set_fixed(h, r < 0 ? -2 : r, type, fixed);
}
int cpm_set_stickiness(cpm_handle* h, int type, int other, float S) {
  return set_stickiness(h, -1, type, other, S);
}
int cpm_set_stickiness_r(cpm_handle* h, int r, int type, int other, float S) {
  return set_stickiness(h, r < 0 ? -2 : r, type, other, S);
}
int cpm_set_adhesion(cpm_handle* h, int type, int other, float J, int symmetric) {
  return set_adhesion(h, -1, type, other, J, symmetric);
}
int cpm_set_adhesion_r(cpm_handle* h, int r, int type, int other, float J, int symmetric) {
  return set_adhesion(h, r < 0 ? -2 : r, type, other, J, symmetric);
}

int cpm_add_cell(cpm_handle* h, int type, int x, int y, int z) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  const DevReplica& R = h->reps[0];
  if (h->ndim == 2) z = 0;
  if (x < 0 || x >= R.nx || y < 0 || y >= R.ny || z < 0 || z >= R.nz)
    return h->fail(CPM_ERR_INVALID, "add_cell position (%d, %d, %d) outside the lattice", x, y, z);
  if (h->added_cells >= R.ncells)
    return h->fail(CPM_ERR_INVALID, "add_cell would exceed number_of_cells = %d", R.ncells);
  h->added_cells += 1;
  h->h_lat[R.lat_off + ((long long)z * R.ny + y) * R.nx + x] =
      (uint32_t)h->added_cells | ((uint32_t)type << 24);
  return CPM_OK;
}

int cpm_host_field_r(cpm_handle* h, int r, double** ptr, int64_t* nvalues) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  if (!h->d_field) {
    const size_t n = (size_t)h->total_sites * h->ndim;
    try {
      h->h_field.assign(n, 0.0);
    } catch (...) {
      return h->fail(CPM_ERR_ALLOC, "host field allocation failed");
    }
    CPM_CUDA(h, cudaMalloc((void**)&h->d_field, sizeof(float) * (n ? n : 1)));
    CPM_CUDA(h, cudaMemsetAsync(h->d_field, 0, sizeof(float) * (n ? n : 1), h->stream));
    if (h->graph_exec) {  // captured without a field
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
  }
  const DevReplica& R = h->reps[r];
  if (ptr) *ptr = h->h_field.data() + (size_t)h->ndim * R.lat_off;
  if (nvalues) *nvalues = (int64_t)h->ndim * R.nx * R.ny * R.nz;
  return CPM_OK;
}

namespace {
int set_act(cpm_handle* h, int r, int type, int max_act, float lambda) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  if (!std::isfinite(lambda)) return h->fail(CPM_ERR_INVALID, "lambda must be finite");
  if (max_act < 0) return h->fail(CPM_ERR_INVALID, "max_act must be >= 0");
  return for_replicas(h, r, [&](DevParams& p) {
    p.act_max[type] = max_act;
    p.act_lambda[type] = lambda;
  });
}

int set_persistence(cpm_handle* h, int r, int type, int time, float diffusion, float lambda) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  if (!std::isfinite(lambda) || !std::isfinite(diffusion))
    return h->fail(CPM_ERR_INVALID, "lambda and diffusion must be finite");
  return for_replicas(h, r, [&](DevParams& p) {
    p.persist_lambda[type] = lambda;
    p.persist_diff[type] = diffusion;
    p.persist_time[type] = time;
  });
}

int set_chemotaxis(cpm_handle* h, int r, int type, float lambda) {
  if (!h) return CPM_ERR_INVALID;
  if (int rc = check_type(h, type)) return rc;
  if (!std::isfinite(lambda)) return h->fail(CPM_ERR_INVALID, "lambda must be finite");
  return for_replicas(h, r, [&](DevParams& p) { p.chemo[type] = lambda; });
}
}  // namespace
int cpm_host_act_r(cpm_handle* h, int r, uint32_t** ptr, int64_t* nsites) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  if (int rc = ensure_act(h)) return rc;
  const DevReplica& R = h->reps[r];
  if (ptr) *ptr = h->h_act.data() + R.lat_off;
  if (nsites) *nsites = (int64_t)R.nx * R.ny * R.nz;
  return CPM_OK;
}
int cpm_has_act(const cpm_handle* h, int* has) {
  if (!h || !has) return CPM_ERR_INVALID;
  *has = h->d_act ? 1 : 0;
  return CPM_OK;
}
int cpm_set_act(cpm_handle* h, int type, int max_act, float lambda) {
  return set_act(h, -1, type, max_act, lambda);
}
int cpm_set_act_r(cpm_handle* h, int r, int type, int max_act, float lambda) {
  return set_act(h, r < 0 ? -2 : r, type, max_act, lambda);
}
int cpm_set_chemotaxis(cpm_handle* h, int type, float lambda) {
  return set_chemotaxis(h, -1, type, lambda);
}
int cpm_set_chemotaxis_r(cpm_handle* h, int r, int type, float lambda) {
  return set_chemotaxis(h, r < 0 ? -2 : r, type, lambda);
}
int cpm_set_persistence(cpm_handle* h, int type, int time, float diffusion, float lambda) {
  return set_persistence(h, -1, type, time, diffusion, lambda);
}
int cpm_set_persistence_r(cpm_handle* h, int r, int type, int time, float diffusion,
                          float lambda) {
  return set_persistence(h, r < 0 ? -2 : r, type, time, diffusion, lambda);
}

int cpm_set_history(cpm_handle* h, int history) {
  if (!h) return CPM_ERR_INVALID;
  if (history < 1) return h->fail(CPM_ERR_INVALID, "history must be >= 1");
  if (history == h->hist_size) return CPM_OK;
  CPM_BIND(h);
  h->hist_size = history;
  if (h->d_hist) {  // reallocated and refilled from the current tables
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree(h->d_hist);
    h->d_hist = nullptr;
    return ensure_persist(h);
  }
  return CPM_OK;
}

int cpm_has_persistence(const cpm_handle* h, int* has, int* history) {
  if (!h) return CPM_ERR_INVALID;
  if (has) *has = (h->d_prefdir && h->d_hist) ? 1 : 0;
  if (history) *history = h->hist_size;
  return CPM_OK;
}

namespace {
// Copies of replica r's rows of the persistence state; `to_host` picks the
// direction.  History slots in the caller's buffer run oldest first.
int persistence_copy(cpm_handle* h, int r, double* prefdir, double* history, bool to_host) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  if (!to_host && h->ndim == 3 && h->pushed) {  // restoring: allocate first
    if (int rc = ensure_persist(h)) return rc;
  }
  if (!h->d_prefdir || !h->d_hist)
    return h->fail(CPM_ERR_STATE, "the engine has no persistence state");
  const DevReplica& R = h->reps[r];
  const size_t n = (size_t)(R.ncells + 1) * 3;
  const auto kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  auto copy = [&](double* dev, double* host) {
    return to_host ? cudaMemcpyAsync(host, dev, n * sizeof(double), kind, h->stream)
                   : cudaMemcpyAsync(dev, host, n * sizeof(double), kind, h->stream);
  };
  if (prefdir) CPM_CUDA(h, copy(h->d_prefdir + R.cell_off * 3, prefdir));
  if (history)
    for (int k = 0; k < h->hist_size; ++k) {
      const int slot = (h->hist_slot + k) % h->hist_size;
      CPM_CUDA(h, copy(h->d_hist + ((size_t)slot * h->rows + R.cell_off) * 3, history + k * n));
    }
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  return CPM_OK;
}
}  // namespace

int cpm_get_persistence_r(cpm_handle* h, int r, double* prefdir, double* history) {
  return persistence_copy(h, r, prefdir, history, true);
}
int cpm_set_persistence_state_r(cpm_handle* h, int r, const double* prefdir,
                                const double* history) {
  return persistence_copy(h, r, const_cast<double*>(prefdir), const_cast<double*>(history),
                          false);
}

int cpm_host_lattice_r(cpm_handle* h, int r, uint32_t** ptr, int64_t* nsites) {
  if (int rc = check_replica(h, r)) return rc;
  const DevReplica& R = h->reps[r];
  if (ptr) *ptr = h->h_lat + R.lat_off;
  if (nsites) *nsites = (int64_t)R.nx * R.ny * R.nz;
  return CPM_OK;
}
int cpm_host_lattice(cpm_handle* h, uint32_t** ptr, int64_t* nsites) {
  return cpm_host_lattice_r(h, 0, ptr, nsites);
}

int cpm_device_lattice_r(cpm_handle* h, int r, uint32_t** dptr) {
  if (int rc = check_replica(h, r)) return rc;
  if (dptr) *dptr = h->d_lat + h->reps[r].lat_off;
  return CPM_OK;
}

namespace {
// Tables of every replica recomputed from the device lattice.
int recount_tables(cpm_handle* h) {
  h->pushed = false;
  for (int b = 0; b < 2; ++b) {
    CPM_CUDA(h, cudaMemsetAsync(h->d_ap[b], 0, sizeof(unsigned long long) * h->rows, h->stream));
    CPM_CUDA(h, cudaMemsetAsync(h->d_cs[b], 0, sizeof(long long) * h->rows * h->ndim, h->stream));
    CPM_CUDA(h, cudaMemsetAsync(h->d_dap[b], 0, sizeof(unsigned long long) * h->rows, h->stream));
    CPM_CUDA(h, cudaMemsetAsync(h->d_dcs[b], 0, sizeof(long long) * h->rows * h->ndim, h->stream));
  }
  CPM_CUDA(h, cudaMemsetAsync(h->d_first, 0xFF, sizeof(unsigned long long) * h->rows, h->stream));
  CPM_CUDA(h, cudaMemsetAsync(h->d_ctype, 0xFF, sizeof(int) * h->rows, h->stream));
  CPM_CUDA(h, cudaMemsetAsync(h->d_ctl, 0, sizeof(uint32_t) * kCtlWords, h->stream));
  CPM_CUDA(h, launch_init(h->ndim, h->d_lat, h->d_reps, h->nrep, h->total_sites,
                          h->d_ap[0], h->d_cs[0], h->d_first, h->d_ctype, h->d_ctl,
                          h->stream));
  h->launches += 2;
  // Both table copies start equal (the sweep keeps them equal between runs).
  CPM_CUDA(h, cudaMemcpyAsync(h->d_ap[1], h->d_ap[0], sizeof(unsigned long long) * h->rows,
                              cudaMemcpyDeviceToDevice, h->stream));
  CPM_CUDA(h, cudaMemcpyAsync(h->d_cs[1], h->d_cs[0], sizeof(long long) * h->rows * h->ndim,
                              cudaMemcpyDeviceToDevice, h->stream));
  uint32_t w = 0;
  if (int rc = read_error_word(h, &w)) return rc;
  if (w) {
    CPM_CUDA(h, cudaMemsetAsync(h->d_ctl, 0, sizeof(uint32_t) * kCtlWords, h->stream));
    return h->fail(CPM_ERR_INVALID, "the lattice was rejected: %s",
                   describe_errors(w).c_str());
  }
  h->pushed = true;
  return CPM_OK;
}
}  // namespace

int cpm_push(cpm_handle* h) {
  CPM_BIND(h);
  h->pushed = false;
  CPM_CUDA(h, cudaMemcpyAsync(h->d_lat, h->h_lat, sizeof(uint32_t) * h->total_sites,
                              cudaMemcpyHostToDevice, h->stream));
  if (h->d_act)  // act stamps go along (src/cpm.cu:547-549)
    CPM_CUDA(h, cudaMemcpyAsync(h->d_act, h->h_act.data(), sizeof(uint32_t) * h->total_sites,
                                cudaMemcpyHostToDevice, h->stream));
  if (h->d_field) {  // the field goes along, as in Cpm::moveCellIdsToGpu
    std::vector<float> f(h->h_field.begin(), h->h_field.end());
    CPM_CUDA(h, cudaMemcpyAsync(h->d_field, f.data(), sizeof(float) * f.size(),
                                cudaMemcpyHostToDevice, h->stream));
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));  // `f` lives on this frame
  }
  if (int rc = recount_tables(h)) return rc;
  if (h->d_hist) {  // every history slot holds the pushed means (src/cpm.cu:578-583)
    CPM_CUDA(h, launch_persist_fill(h->d_hist, h->hist_size, h->d_ap[0], h->d_cs[0], h->d_reps,
                                    h->nrep, h->rows, h->stream));
    h->hist_slot = 0;
  }
  return CPM_OK;
}

int cpm_recount(cpm_handle* h) {
  CPM_BIND(h);
  return recount_tables(h);
}

int cpm_set_centroid_sums_r(cpm_handle* h, int r, const int64_t* centroid_sums) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  if (!centroid_sums) return h->fail(CPM_ERR_INVALID, "centroid_sums is NULL");
  if (!h->pushed) return h->fail(CPM_ERR_STATE, "set centroid sums after a successful push");
  const DevReplica& R = h->reps[r];
  const size_t bytes = sizeof(long long) * ((size_t)R.ncells + 1) * h->ndim;
  for (int b = 0; b < 2; ++b)
    CPM_CUDA(h, cudaMemcpyAsync(h->d_cs[b] + R.cell_off * h->ndim, centroid_sums, bytes,
                                cudaMemcpyHostToDevice, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));  // the caller's buffer may go
  return CPM_OK;
}

int cpm_get_params_r(const cpm_handle* h, int r, cpm_static_params* out) {
  if (!h || !out || r < 0 || r >= h->nrep) return CPM_ERR_INVALID;
  const DevParams& p = h->psets[h->reps[r].pset];
  std::memcpy(out->J, p.J, sizeof out->J);
  std::memcpy(out->lambda_area, p.lam_area, sizeof out->lambda_area);
  std::memcpy(out->target_area, p.tgt_area, sizeof out->target_area);
  std::memcpy(out->lambda_perimeter, p.lam_perim, sizeof out->lambda_perimeter);
  std::memcpy(out->target_perimeter, p.tgt_perim, sizeof out->target_perimeter);
  out->temperature = p.temperature;
  std::memcpy(out->stickiness, p.stick, sizeof out->stickiness);
  for (int k = 0; k < kMaxTypes; ++k) out->fixed[k] = (p.fixed_mask >> k) & 1u;
  std::memcpy(out->chemotaxis, p.chemo, sizeof out->chemotaxis);
  std::memcpy(out->act_lambda, p.act_lambda, sizeof out->act_lambda);
  std::memcpy(out->act_max, p.act_max, sizeof out->act_max);
  std::memcpy(out->persistence_lambda, p.persist_lambda, sizeof out->persistence_lambda);
  std::memcpy(out->persistence_diffusion, p.persist_diff, sizeof out->persistence_diffusion);
  std::memcpy(out->persistence_time, p.persist_time, sizeof out->persistence_time);
  return CPM_OK;
}

namespace {
int set_params(cpm_handle* h, int r, const cpm_static_params* in) {
  if (!h) return CPM_ERR_INVALID;
  if (!in) return h->fail(CPM_ERR_INVALID, "params is NULL");
  if (!std::isfinite(in->temperature))
    return h->fail(CPM_ERR_INVALID, "temperature must be finite");
  for (int k = 0; k < kMaxTypes; ++k) {
    if (!std::isfinite(in->chemotaxis[k]) || !std::isfinite(in->act_lambda[k]) ||
        !std::isfinite(in->persistence_lambda[k]) || !std::isfinite(in->persistence_diffusion[k]))
      return h->fail(CPM_ERR_INVALID, "lambdas and diffusion must be finite");
    if (in->act_max[k] < 0) return h->fail(CPM_ERR_INVALID, "act_max must be >= 0");
  }
  auto fill = [&](DevParams& p) {
    std::memcpy(p.J, in->J, sizeof p.J);
    std::memcpy(p.lam_area, in->lambda_area, sizeof p.lam_area);
    std::memcpy(p.tgt_area, in->target_area, sizeof p.tgt_area);
    std::memcpy(p.lam_perim, in->lambda_perimeter, sizeof p.lam_perim);
    std::memcpy(p.tgt_perim, in->target_perimeter, sizeof p.tgt_perim);
    p.temperature = in->temperature;
    std::memcpy(p.stick, in->stickiness, sizeof p.stick);
    p.fixed_mask = 0;
    for (int k = 0; k < kMaxTypes; ++k)
      if (in->fixed[k]) p.fixed_mask |= 1u << k;
    std::memcpy(p.chemo, in->chemotaxis, sizeof p.chemo);
    std::memcpy(p.act_lambda, in->act_lambda, sizeof p.act_lambda);
    std::memcpy(p.act_max, in->act_max, sizeof p.act_max);
    std::memcpy(p.persist_lambda, in->persistence_lambda, sizeof p.persist_lambda);
    std::memcpy(p.persist_diff, in->persistence_diffusion, sizeof p.persist_diff);
    std::memcpy(p.persist_time, in->persistence_time, sizeof p.persist_time);
  };
  if (r == -1) {  // every field of every replica: one shared record
    DevParams p;
    default_params(p, in->temperature);
    fill(p);
    h->psets.assign(1, p);
    h->pset_refs.assign(1, h->nrep);
    for (auto& R : h->reps) R.pset = 0;
    h->reps_dirty = true;
    h->params_dirty = true;
    return CPM_OK;
  }
  return for_replicas(h, r, fill);
}
}  // namespace

int cpm_set_params(cpm_handle* h, const cpm_static_params* in) { return set_params(h, -1, in); }
int cpm_set_params_r(cpm_handle* h, int r, const cpm_static_params* in) {
  return set_params(h, r < 0 ? -2 : r, in);
}

int cpm_get_param_index(const cpm_handle* h, int* out) {
  if (!h || !out) return CPM_ERR_INVALID;
  for (int r = 0; r < h->nrep; ++r) out[r] = h->reps[r].pset;
  return CPM_OK;
}

int cpm_get_device(const cpm_handle* h, int* device) {
  if (!h || !device) return CPM_ERR_INVALID;
  *device = h->device;
  return CPM_OK;
}

int cpm_get_seed(const cpm_handle* h, uint64_t* seed, uint32_t* stream_id) {
  if (!h) return CPM_ERR_INVALID;
  if (seed) *seed = h->seed;
  if (stream_id) *stream_id = h->stream_id;
  return CPM_OK;
}

int cpm_pull(cpm_handle* h) {
  CPM_BIND(h);
  CPM_CUDA(h, cudaMemcpyAsync(h->h_lat, h->d_lat, sizeof(uint32_t) * h->total_sites,
                              cudaMemcpyDeviceToHost, h->stream));
  if (h->d_act)  // and the act stamps (src/cpm.cu:534-536)
    CPM_CUDA(h, cudaMemcpyAsync(h->h_act.data(), h->d_act, sizeof(uint32_t) * h->total_sites,
                                cudaMemcpyDeviceToHost, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  return CPM_OK;
}

int cpm_run(cpm_handle* h, int mcs) {
  CPM_BIND(h);
  if (mcs < 0) return h->fail(CPM_ERR_INVALID, "mcs must be >= 0");
  if (!h->pushed) return h->fail(CPM_ERR_STATE, "run() before a successful push_to_gpu()");
  if (mcs == 0) return CPM_OK;
  if (int rc = upload_params(h)) return rc;
  SweepArgs a = sweep_args(h, run_variant(h));
  int left = mcs;
  while (left > 0) {
    const int chunk = std::min(left, kMaxMcsPerLaunch);
    a.tick0 = h->tick;
    a.mcs = chunk;
    // The barrier counter starts at zero in every launch; the sticky error
    // word is left alone until cpm_synchronize reads it.
    int nl = 0;
    CPM_CUDA(h, enqueue_sweep(h, run_variant(h), h->dispatch, a, false, &nl));
    h->launches += nl;
    h->tick += (uint64_t)chunk;
    left -= chunk;
  }
  h->d_tick_stale = true;
  count_attempts(h, mcs);
  return persist_after_run(h);
}

int cpm_run_graph(cpm_handle* h, int mcs) {
  CPM_BIND(h);
  if (mcs <= 0 || mcs > kMaxMcsPerLaunch)
    return h->fail(CPM_ERR_INVALID, "mcs must be in [1, %d] for a graph run", kMaxMcsPerLaunch);
  if (!h->pushed) return h->fail(CPM_ERR_STATE, "run before a successful push_to_gpu()");
  if (h->stream == nullptr)
    return h->fail(CPM_ERR_STATE, "graph runs need a non-default stream");
  if (int rc = upload_params(h)) return rc;
  if (!h->graph_exec || h->graph_mcs != mcs || h->graph_variant != run_variant(h) ||
      h->graph_dispatch != h->dispatch || h->graph_fill != fill_key(h) ||
      h->graph_stream != h->stream) {
    if (h->graph_exec) {
      cudaGraphExecDestroy(h->graph_exec);
      h->graph_exec = nullptr;
    }
    // Capture: reset the barrier words, then the persistent sweep reading
    // its start time from (and advancing) the device tick.
    SweepArgs a = sweep_args(h, run_variant(h));
    a.tick_ptr = h->d_tick;
    a.mcs = mcs;
    cudaGraph_t g = nullptr;
    CPM_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int nl = 0;
    cudaError_t e2 = enqueue_sweep(h, run_variant(h), h->dispatch, a, false, &nl);
    cudaError_t e3 = cudaStreamEndCapture(h->stream, &g);
    if (e2 != cudaSuccess) return h->cuda_fail(e2, "capture of the sweep launch");
    if (e3 != cudaSuccess) return h->cuda_fail(e3, "cudaStreamEndCapture");
    cudaError_t e4 = cudaGraphInstantiate(&h->graph_exec, g, 0);
    cudaGraphDestroy(g);
    if (e4 != cudaSuccess) return h->cuda_fail(e4, "cudaGraphInstantiate");
    h->graph_mcs = mcs;
    h->graph_launches = nl;
    h->graph_variant = run_variant(h);
    h->graph_dispatch = h->dispatch;
    h->graph_fill = fill_key(h);
    h->graph_stream = h->stream;
  }
  if (h->d_tick_stale) {
    const unsigned long long t = h->tick;
    CPM_CUDA(h, cudaMemcpyAsync(h->d_tick, &t, sizeof t, cudaMemcpyHostToDevice, h->stream));
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));  // `t` lives on this frame
    h->d_tick_stale = false;
  }
  CPM_CUDA(h, cudaGraphLaunch(h->graph_exec, h->stream));
  h->launches += h->graph_launches;
  h->tick += (uint64_t)mcs;
  count_attempts(h, mcs);
  return persist_after_run(h);  // a launch of its own: its slot changes per run
}

int cpm_autotune(cpm_handle* h, int probe_mcs, int* chosen, float* ms_per_mcs) {
  CPM_BIND(h);
  if (!h->pushed) return h->fail(CPM_ERR_STATE, "autotune before a successful push_to_gpu()");
  if (probe_mcs < 1) probe_mcs = 2;
  if (int rc = upload_params(h)) return rc;
  // Work on a saved copy of the state: every variant runs the same MCS from
  // the same start, and the state (lattice, tables, counters, tick) is put
  // back afterwards.  The sweep's result does not depend on the variant, so
  // only the time differs.
  const size_t lat_b = sizeof(uint32_t) * h->total_sites;
  const size_t ap_b = sizeof(unsigned long long) * h->rows;
  const size_t cs_b = sizeof(long long) * h->rows * h->ndim;
  const size_t cnt_b = sizeof(unsigned long long) * 2 * h->nrep;
  const size_t act_b = h->d_act ? lat_b : 0;  // act stamps, when kept
  char* save = nullptr;
  CPM_CUDA(h, cudaMalloc(&save, lat_b + ap_b + cs_b + cnt_b + act_b));
  auto copy = [&](bool to_save) -> cudaError_t {
    char* p = save;
    void* dst[5] = {p, p + lat_b, p + lat_b + ap_b, p + lat_b + ap_b + cs_b,
                    p + lat_b + ap_b + cs_b + cnt_b};
    void* src[5] = {h->d_lat, h->d_ap[0], h->d_cs[0], h->d_counters, h->d_act};
    const size_t n[5] = {lat_b, ap_b, cs_b, cnt_b, act_b};
    for (int i = 0; i < 5; ++i) {
      if (!n[i]) continue;
      cudaError_t e = to_save ? cudaMemcpyAsync(dst[i], src[i], n[i], cudaMemcpyDeviceToDevice, h->stream)
                              : cudaMemcpyAsync(src[i], dst[i], n[i], cudaMemcpyDeviceToDevice, h->stream);
      if (e != cudaSuccess) return e;
    }
    if (!to_save) {
      cudaError_t e = cudaMemcpyAsync(h->d_ap[1], h->d_ap[0], ap_b, cudaMemcpyDeviceToDevice, h->stream);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(h->d_cs[1], h->d_cs[0], cs_b, cudaMemcpyDeviceToDevice, h->stream);
      return e;
    }
    return cudaSuccess;
  };
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaError_t e = cudaEventCreate(&ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
  if (e == cudaSuccess) e = copy(true);
  const uint64_t tick = h->tick;
  float best = -1.0f;
  int best_v = run_variant(h), best_d = h->dispatch;
  // Every (tile variant, dispatch) pair, replica dispatch only for batches,
  // timed in three rounds (the fastest run counts): a variant's first launch
  // also loads its module, and clocks may still be rising.
  // (hybrid only where it splits the batch into two non-empty parts)
  std::vector<std::pair<int, int>> pairs;
  for (int d = 0; d < (h->nrep > 1 ? 3 : 1); ++d)
    for (int v = 0; v < kTileVariants; ++v)
      if (d != CPM_DISPATCH_HYBRID || (h->cfg[v].hyb_ng > 0 && h->cfg[v].hyb_ng < h->nrep))
        pairs.emplace_back(v, d);
  // A lattice that one thread-block cluster can hold is also tried in the
  // cluster sweep (which has no tile variants), unless the caller chose the
  // parity fill.  Runs with the act or persistence term never take it: the fill
  // stays as it is then, as after an error.
  const int row_fill = h->fill != CPM_FILL_CLUSTER ? h->fill
                       : h->row_ok                 ? CPM_FILL_TMA
                                                   : CPM_FILL_PARITY;
  const auto fill_by = h->fill_by;
  const int fill = h->fill;
  const bool try_cluster = h->cluster_blocks > 0 && !h->act_active && !h->persist_active &&
                           (fill_by == cpm_handle::kBySize || fill != CPM_FILL_PARITY);
  if (try_cluster) pairs.emplace_back(run_variant(h), -1);
  h->fill_by = cpm_handle::kByTuner;
  int best_fill = row_fill;
  const int npairs = (int)pairs.size();
  for (int i = 0; i < 3 * npairs && e == cudaSuccess; ++i) {
    const int v = pairs[i % npairs].first;
    const bool cl = pairs[i % npairs].second < 0;
    const int d = cl ? CPM_DISPATCH_GRID : pairs[i % npairs].second;
    h->fill = cl ? CPM_FILL_CLUSTER : row_fill;
    SweepArgs a = sweep_args(h, v);
    a.tick0 = tick;
    a.mcs = probe_mcs;
    e = copy(false);
    if (e == cudaSuccess) e = cudaEventRecord(ev[0], h->stream);
    int nl = 0;
    if (e == cudaSuccess) e = enqueue_sweep(h, v, d, a, false, &nl);
    if (e == cudaSuccess) e = cudaEventRecord(ev[1], h->stream);
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
    float ms = 0.0f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ev[0], ev[1]);
    h->launches += nl;
    if (e == cudaSuccess && (best < 0.0f || ms < best)) {
      best = ms;
      best_v = v;
      best_d = d;
      best_fill = h->fill;
    }
  }
  h->fill = fill;
  h->fill_by = fill_by;
  if (e == cudaSuccess) e = copy(false);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(save);
  if (ev[0]) cudaEventDestroy(ev[0]);
  if (ev[1]) cudaEventDestroy(ev[1]);
  if (e != cudaSuccess) return h->cuda_fail(e, "autotune");
  uint32_t w = 0;
  if (int rc = read_error_word(h, &w)) return rc;
  if (w) return h->fail(CPM_ERR_TIMEOUT, "autotune: %s", describe_errors(w).c_str());
  h->variant = best_v;
  h->variant_ext = h->act_active || h->persist_active;
  h->dispatch = best_d;
  if (try_cluster && (fill_by == cpm_handle::kBySize || best_fill != fill ||
                      best_fill == CPM_FILL_CLUSTER)) {
    h->fill = best_fill;
    h->fill_by = cpm_handle::kByTuner;
  }
  h->tick = tick;
  if (chosen) *chosen = best_v;
  if (ms_per_mcs) *ms_per_mcs = best / (float)probe_mcs;
  return CPM_OK;
}

static_assert(sizeof(cpm_score_spec) == sizeof(ScoreSpec), "score spec layout");
static_assert(CPM_SCORE_MAX == kScoreMax, "score width");

int cpm_run_scores(cpm_handle* h, int mcs, float* d_scores, uint64_t score_base,
                   int score_len, const cpm_score_spec* spec) {
  CPM_BIND(h);
  if (h->ndim != 2) return h->fail(CPM_ERR_UNSUPPORTED, "scores are computed for 2D engines");
  if (mcs < 0 || !d_scores || !spec || score_len < 0)
    return h->fail(CPM_ERR_INVALID, "cpm_run_scores: bad arguments");
  if (!h->pushed) return h->fail(CPM_ERR_STATE, "run before a successful push_to_gpu()");
  ScoreSpec sp;
  std::memcpy(&sp, spec, sizeof sp);
  if (sp.n_pairs < 0 || sp.n_pairs > kScorePairsMax ||
      sp.n_pairs + (sp.lambda_area ? 1 : 0) + (sp.lambda_perim ? 1 : 0) +
              (sp.temperature ? 1 : 0) > kScoreMax)
    return h->fail(CPM_ERR_INVALID, "cpm_run_scores: too many score parameters");
  for (int k = 0; k < sp.n_pairs; ++k)
    if (sp.pair_a[k] < 0 || sp.pair_a[k] >= kScoreTypes || sp.pair_b[k] < 0 ||
        sp.pair_b[k] >= kScoreTypes)
      return h->fail(CPM_ERR_INVALID, "cpm_run_scores: score types must be < %d", kScoreTypes);
  if (mcs == 0) return CPM_OK;
  if (int rc = upload_params(h)) return rc;
  if (h->act_active || h->persist_active)
    return h->fail(CPM_ERR_UNSUPPORTED, "cpm_run_scores: scores of runs with the act or "
                                        "persistence term are not supported");
  SweepArgs a = sweep_args(h, run_variant(h));
  a.scores = d_scores;
  a.score_base = score_base;
  a.score_len = score_len;
  a.score_spec = sp;
  int left = mcs;
  while (left > 0) {
    const int chunk = std::min(left, kMaxMcsPerLaunch);
    a.tick0 = h->tick;
    a.mcs = chunk;
    int nl = 0;
    CPM_CUDA(h, enqueue_sweep(h, run_variant(h), h->dispatch, a, true, &nl));
    h->launches += nl;
    h->tick += (uint64_t)chunk;
    left -= chunk;
  }
  h->d_tick_stale = true;
  count_attempts(h, mcs);
  return CPM_OK;
}

int cpm_observe_heterotypic(cpm_handle* h, float* out_host) {
  CPM_BIND(h);
  if (h->ndim != 2) return h->fail(CPM_ERR_UNSUPPORTED, "2D engines only");
  if (!out_host) return h->fail(CPM_ERR_INVALID, "out_host is NULL");
  // [nrep + 1] first tasks, then [2 nrep] counts, in one buffer
  std::vector<long long> start(h->nrep + 1, 0);
  for (int r = 0; r < h->nrep; ++r) {
    const DevReplica& R = h->reps[r];
    start[r + 1] = start[r] + ((R.nx + 31LL) / 32) * ((R.ny + kObserveRows - 1LL) / kObserveRows);
  }
  const size_t start_b = sizeof(long long) * (h->nrep + 1),
               counts_b = sizeof(unsigned long long) * 2 * h->nrep;
  if (int rc = ensure_scratch(h, start_b + counts_b)) return rc;
  char* buf = h->d_scratch;
  unsigned long long* counts = reinterpret_cast<unsigned long long*>(buf + start_b);
  cudaError_t e = cudaMemcpyAsync(buf, start.data(), start_b, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(counts, 0, counts_b, h->stream);
  if (e == cudaSuccess)
    e = launch_observe_heterotypic(h->d_lat, h->d_reps, h->nrep,
                                   reinterpret_cast<const long long*>(buf), start[h->nrep],
                                   counts, h->stream);
  h->launches += 1;
  std::vector<unsigned long long> c(2 * h->nrep);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(c.data(), counts, counts_b, cudaMemcpyDeviceToHost, h->stream);
  // (also on an error: the copies read and write this frame's vectors)
  const cudaError_t e2 = cudaStreamSynchronize(h->stream);
  trim_scratch(h);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return h->cuda_fail(e, "cpm_observe_heterotypic");
  for (int r = 0; r < h->nrep; ++r)
    out_host[r] = c[2 * r] ? (float)((double)c[2 * r + 1] / (double)c[2 * r]) : 0.0f;
  return CPM_OK;
}

int cpm_seed_voronoi_r(cpm_handle* h, int r, int npoints, const double* points,
                       const uint32_t* values) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  if (npoints < 1 || !points || !values)
    return h->fail(CPM_ERR_INVALID, "cpm_seed_voronoi_r: need npoints >= 1, points, values");
  const DevReplica& R = h->reps[r];
  const int nd = h->ndim;
  const int n[3] = {R.nx, R.ny, R.nz};
  const VoronoiGrid vg = voronoi_grid(nd, n, npoints);
  const double sites = (double)n[0] * n[1] * n[2], wmin = vg.wmin, wmax = vg.wmax;
  const long long G = (long long)vg.g[0] * vg.g[1] * vg.g[2];
  // One pass over the points checks them and finds their buckets (a point at
  // a bucket's edge may be rounded into the next one: the scans allow for it).  The
  // host side of seeding 2048^2 sites from 42,000 points is passes over the
  // points: no divisions, no buffers cleared before they are filled.
  const std::unique_ptr<int[]> bucket_of(new int[npoints]);
  for (int k = 0; k < npoints; ++k) {
    const double* p = points + (size_t)k * nd;
    long long b = 0;
    for (int a = nd - 1; a >= 0; --a) {
      if (!(p[a] >= 0.0 && p[a] < (double)n[a]))
        return h->fail(CPM_ERR_INVALID, "cpm_seed_voronoi_r: point %d lies outside [0, n)", k);
      b = b * vg.g[a] + std::min((int)(p[a] * vg.inv[a]), vg.g[a] - 1);
    }
    bucket_of[k] = (int)b;
    const uint32_t v = values[k], id = v & 0xFFFFFFu, ty = v >> 24;
    if ((int)id > R.ncells || ty >= (uint32_t)kMaxTypes || (id == 0 && ty != 0))
      return h->fail(CPM_ERR_INVALID,
                     "cpm_seed_voronoi_r: value %d is not id <= ncells | type < 32 << 24 "
                     "(id 0 with type 0)", k);
  }
  if (G > (1LL << 30))
    return h->fail(CPM_ERR_INVALID, "cpm_seed_voronoi_r: too many buckets");
  // Counting sort of the points by bucket (host; O(npoints)).
  std::vector<int> start(G + 1, 0);
  for (int k = 0; k < npoints; ++k) ++start[bucket_of[k] + 1];
  for (long long b = 0; b < G; ++b) start[b + 1] += start[b];
  // Work bound.  A site's search ends within about (d + 1) sqrt(ndim)
  // max(w) / min(w) + 1 rings, d the Chebyshev distance (in buckets, wrapped)
  // from its bucket to the nearest occupied one; d comes from a breadth-first
  // search over the bucket grid (its first step from the empty buckets, which
  // are the fewer: of evenly spread points one bucket in eight is empty).
  // Point sets clustered so much that the search would run for seconds are
  // refused instead of launched.
  {
    std::vector<int> dist(G, -1), frontier, next;
    // f(b2) for the wrapped neighbours, until it returns true
    auto neighbours = [&](int b, auto&& f) {
      const int gx = vg.g[0], gy = vg.g[1], gz = vg.g[2];
      const int bx = b % gx, by = (b / gx) % gy, bz = b / (gx * gy);
      auto wrap = [](int i, int g) { return i < 0 ? i + g : (i < g ? i : i - g); };
      for (int dz = (nd == 3 ? -1 : 0); dz <= (nd == 3 ? 1 : 0); ++dz)
        for (int dy = -1; dy <= 1; ++dy) {
          const int row = (wrap(bz + dz, gz) * gy + wrap(by + dy, gy)) * gx;
          for (int dx = -1; dx <= 1; ++dx)
            if (f(row + wrap(bx + dx, gx))) return;
        }
    };
    for (long long b = 0; b < G; ++b)
      if (start[b + 1] > start[b]) dist[b] = 0;
    for (long long b = 0; b < G; ++b) {
      if (dist[b] >= 0) continue;
      bool near = false;
      neighbours((int)b, [&](int b2) { return near = dist[b2] == 0; });
      if (near) frontier.push_back((int)b);
    }
    for (int b : frontier) dist[b] = 1;
    for (int d = 2; !frontier.empty(); ++d) {
      next.clear();
      for (int b : frontier)
        neighbours(b, [&](int b2) {
          if (dist[b2] < 0) {
            dist[b2] = d;
            next.push_back(b2);
          }
          return false;
        });
      frontier.swap(next);
    }
    const double per_bucket_sites = sites / (double)G;
    const double per_bucket_points = (double)npoints / (double)G;
    std::vector<long long> at_dist;  // buckets at each distance
    for (long long b = 0; b < G; ++b) {
      if ((size_t)dist[b] >= at_dist.size()) at_dist.resize(dist[b] + 1, 0);
      ++at_dist[dist[b]];
    }
    double work = 0.0;  // estimated distance evaluations
    for (size_t d = 0; d < at_dist.size(); ++d) {
      const double rings = std::min(
          (double)vg.rmax, ((double)d + 1.0) * std::sqrt((double)nd) * wmax / wmin + 1.0);
      work += (double)at_dist[d] * per_bucket_sites * std::pow(2.0 * rings + 1.0, nd) *
              std::max(1.0, per_bucket_points);
    }
    if (work > 5e11)
      return h->fail(CPM_ERR_INVALID,
                     "cpm_seed_voronoi_r: the points are too unevenly spread for the bucketed "
                     "search (about %.3g distance evaluations); spread them more evenly or "
                     "label the lattice on the host", work);
  }
  // Up go the caller's points and values as they are, and the order of the
  // points by bucket with the buckets' starts; a kernel lays the points out in
  // that order.  (Laid out here, 44 bytes a point in a fresh buffer, they took
  // 0.45 of the 0.88 ms of seeding 2048^2 sites from 42,000 points.)
  const size_t np = (size_t)npoints;
  const size_t off_p = sizeof(float4) * np, off_r = off_p + sizeof(double) * 3 * np,
               off_i = off_r + sizeof(double) * nd * np, off_s = off_i + sizeof(int) * np,
               off_v = off_s + sizeof(int) * (size_t)(G + 1),
               bytes = off_v + sizeof(uint32_t) * np;
  const std::unique_ptr<int[]> up(new int[np + G + 1]);  // order, starts
  std::copy(start.begin(), start.end(), up.get() + np);
  for (int k = 0; k < npoints; ++k) up[start[bucket_of[k]]++] = k;
  if (int rc = ensure_scratch(h, bytes)) return rc;
  char* dev = h->d_scratch;
  cudaError_t e = cudaMemcpyAsync(dev + off_r, points, sizeof(double) * nd * np,
                                  cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dev + off_i, up.get(), off_v - off_i, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dev + off_v, values, sizeof(uint32_t) * np, cudaMemcpyHostToDevice,
                        h->stream);
  if (e == cudaSuccess)
    e = launch_voronoi(h->d_lat + R.lat_off, vg, npoints,
                       reinterpret_cast<const double*>(dev + off_r),
                       reinterpret_cast<double*>(dev + off_p), reinterpret_cast<float4*>(dev),
                       reinterpret_cast<const int*>(dev + off_i),
                       reinterpret_cast<const uint32_t*>(dev + off_v),
                       reinterpret_cast<const int*>(dev + off_s), h->stream);
  h->launches += 2;
  // the host buffers are read by the copies: wait before they go
  const cudaError_t e2 = cudaStreamSynchronize(h->stream);
  trim_scratch(h);
  if (e != cudaSuccess) return h->cuda_fail(e, "cpm_seed_voronoi_r");
  if (e2 != cudaSuccess) return h->cuda_fail(e2, "cpm_seed_voronoi_r");
  h->pushed = false;  // the tables no longer describe the lattice
  return CPM_OK;
}

int cpm_observe_boundaries(cpm_handle* h, int ntypes, uint64_t* out_host) {
  CPM_BIND(h);
  if (ntypes < 1 || ntypes > kMaxTypes)
    return h->fail(CPM_ERR_INVALID, "ntypes must be in [1, %d]", kMaxTypes);
  if (!out_host) return h->fail(CPM_ERR_INVALID, "out_host is NULL");
  std::vector<long long> tile_start(h->nrep + 1, 0);
  for (int r = 0; r < h->nrep; ++r) {
    const DevReplica& R = h->reps[r];
    const long long sites = (long long)R.nx * R.ny * R.nz;
    tile_start[r + 1] = tile_start[r] + (sites + kBoundaryTile - 1) / kBoundaryTile;
  }
  const long long ntiles = tile_start[h->nrep];
  const size_t nc = (size_t)h->nrep * ntypes * ntypes;
  const size_t ts_b = sizeof(long long) * (h->nrep + 1), counts_b = sizeof(uint64_t) * nc;
  if (int rc = ensure_scratch(h, ts_b + counts_b)) return rc;
  long long* d_ts = reinterpret_cast<long long*>(h->d_scratch);
  unsigned long long* counts = reinterpret_cast<unsigned long long*>(h->d_scratch + ts_b);
  cudaError_t e = cudaMemsetAsync(counts, 0, counts_b, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_ts, tile_start.data(), ts_b, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = launch_observe_boundaries(h->ndim, h->d_lat, h->d_reps, h->nrep, d_ts, ntiles, ntypes,
                                  counts, h->stream);
  h->launches += 1;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(out_host, counts, counts_b, cudaMemcpyDeviceToHost, h->stream);
  const cudaError_t e2 = cudaStreamSynchronize(h->stream);
  trim_scratch(h);
  if (e != cudaSuccess) return h->cuda_fail(e, "cpm_observe_boundaries");
  if (e2 != cudaSuccess) return h->cuda_fail(e2, "cpm_observe_boundaries");
  return CPM_OK;
}

int cpm_lr_backward(const float* scores, const float* dl_do, const float* obs,
                    const int* checkpoints, int nrep, int len, int nparam, int ncheck,
                    const float* obs_total, int nrep_total, float* grad, void* stream) {
  if (!scores || !dl_do || !obs || !checkpoints || !grad || nrep < 1 || len < 0 ||
      nparam < 1 || nparam > kScoreMax || ncheck < 1 || ncheck > kMaxCheckpoints ||
      (obs_total && nrep_total < nrep)) {
    g_create_error = "cpm_lr_backward: bad arguments";
    return CPM_ERR_INVALID;
  }
  cudaGetLastError();  // (of an earlier call, see CPM_BIND)
  cudaError_t e = launch_lr_backward(scores, dl_do, obs, checkpoints, nrep, len, nparam,
                                     ncheck, obs_total, nrep_total, grad,
                                     (cudaStream_t)stream);
  if (e != cudaSuccess) {
    g_create_error = std::string("cpm_lr_backward: ") + cudaGetErrorString(e);
    return CPM_ERR_CUDA;
  }
  return CPM_OK;
}

int cpm_set_variant(cpm_handle* h, int variant) {
  if (!h) return CPM_ERR_INVALID;
  if (variant < 0 || variant >= kTileVariants)
    return h->fail(CPM_ERR_INVALID, "tile variant %d out of range [0, %d)", variant, kTileVariants);
  h->variant = variant;
  h->variant_ext = false;
  return CPM_OK;
}

int cpm_set_fill(cpm_handle* h, int fill) {
  if (!h) return CPM_ERR_INVALID;
  if (fill != CPM_FILL_PARITY && fill != CPM_FILL_VECTOR && fill != CPM_FILL_TMA &&
      fill != CPM_FILL_CLUSTER)
    return h->fail(CPM_ERR_INVALID, "fill %d is not parity (0), vector (1), tma (2) or "
                                    "cluster (3)", fill);
  if (fill == CPM_FILL_CLUSTER && h->cluster_blocks == 0 && !h->cluster_shape)
    return h->fail(CPM_ERR_UNSUPPORTED, "no thread-block cluster holds this lattice (one 2D "
                                        "lattice, nx from 4 and sides to 4095, that fits the "
                                        "shared memory of 16 or 8 blocks with its tables)");
  if ((fill == CPM_FILL_VECTOR || fill == CPM_FILL_TMA) && !h->row_ok)
    return h->fail(CPM_ERR_UNSUPPORTED, "vector and tma need one lattice with nx a multiple of 4 "
                                        "and nx >= 72; in 2D ny >= 66, in 3D ny, nz >= 18");
  h->fill = fill;
  h->fill_by = cpm_handle::kByCaller;
  return CPM_OK;
}

int cpm_get_fill(const cpm_handle* h, int* fill) {
  if (!h || !fill) return CPM_ERR_INVALID;
  *fill = h->fill;
  return CPM_OK;
}

int cpm_running_fill(const cpm_handle* h, int* fill) {
  if (!h || !fill) return CPM_ERR_INVALID;
  if (uses_cluster(h))
    *fill = CPM_FILL_CLUSTER;
  else
    *fill = h->fill_by == cpm_handle::kByCaller && h->fill != CPM_FILL_CLUSTER ? h->fill
                                                                              : CPM_FILL_PARITY;
  return CPM_OK;
}

int cpm_set_dispatch(cpm_handle* h, int dispatch) {
  if (!h) return CPM_ERR_INVALID;
  if (dispatch != CPM_DISPATCH_GRID && dispatch != CPM_DISPATCH_REPLICA &&
      dispatch != CPM_DISPATCH_HYBRID)
    return h->fail(CPM_ERR_INVALID, "dispatch %d is not grid (0), replica (1) or hybrid (2)",
                   dispatch);
  if (dispatch != CPM_DISPATCH_GRID && h->nrep < 2)
    return h->fail(CPM_ERR_UNSUPPORTED, "replica and hybrid dispatch need a batch of two or "
                                        "more replicas");
  h->dispatch = dispatch;
  return CPM_OK;
}

int cpm_synchronize(cpm_handle* h) {
  CPM_BIND(h);
  uint32_t w = 0;
  if (int rc = read_error_word(h, &w)) return rc;
  if (w) {
    CPM_CUDA(h, cudaMemsetAsync(h->d_ctl + kCtlErr, 0, sizeof(uint32_t), h->stream));
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
    h->pushed = false;  // the lattice and tables may disagree now
    return h->fail((w & kErrTimeout) ? CPM_ERR_TIMEOUT : CPM_ERR_INVALID,
                   "sweep failed: %s", describe_errors(w).c_str());
  }
  return CPM_OK;
}

int cpm_set_stream(cpm_handle* h, void* stream) {
  CPM_BIND(h);
  cudaStream_t next = stream ? (cudaStream_t)stream : h->own_stream;
  if (next != h->stream) {
    // Work already queued on the old stream must finish before the new one
    // touches the same buffers.
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
    h->stream = next;
  }
  return CPM_OK;
}

int cpm_set_seed(cpm_handle* h, uint64_t seed, uint32_t stream_id) {
  if (!h) return CPM_ERR_INVALID;
  h->seed = seed;
  h->stream_id = stream_id;
  return CPM_OK;
}

int cpm_get_tick(const cpm_handle* h, uint64_t* tick) {
  if (!h || !tick) return CPM_ERR_INVALID;
  *tick = h->tick;
  return CPM_OK;
}

int cpm_set_tick(cpm_handle* h, uint64_t tick) {
  if (!h) return CPM_ERR_INVALID;
  h->tick = tick;
  h->d_tick_stale = true;
  return CPM_OK;
}

int cpm_get_tables_r(cpm_handle* h, int r, int32_t* area, int32_t* perimeter,
                     int64_t* centroid_sums) {
  if (int rc = check_replica(h, r)) return rc;
  CPM_BIND(h);
  const DevReplica& R = h->reps[r];
  const long long n1 = (long long)R.ncells + 1;
  if (area || perimeter) {
    std::vector<unsigned long long> ap(n1);
    CPM_CUDA(h, cudaMemcpyAsync(ap.data(), h->d_ap[0] + R.cell_off,
                                sizeof(unsigned long long) * n1, cudaMemcpyDeviceToHost,
                                h->stream));
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
    for (long long c = 0; c < n1; ++c) {
      if (area) area[c] = unpack_area(ap[c]);
      if (perimeter) perimeter[c] = unpack_perim(ap[c]);
    }
  }
  if (centroid_sums) {
    CPM_CUDA(h, cudaMemcpyAsync(centroid_sums, h->d_cs[0] + R.cell_off * h->ndim,
                                sizeof(long long) * n1 * h->ndim,
                                cudaMemcpyDeviceToHost, h->stream));
    CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  return CPM_OK;
}

int cpm_get_centroids(cpm_handle* h, double* out, int capacity, int* n_out) {
  CPM_BIND(h);
  const int n = h->added_cells;
  if (n_out) *n_out = n;
  if (!out || capacity <= 0 || n == 0) return CPM_OK;
  const DevReplica& R = h->reps[0];
  const int d = h->ndim;
  const int m = std::min(n, capacity);
  std::vector<unsigned long long> ap(m);
  std::vector<long long> cs((size_t)m * d);
  CPM_CUDA(h, cudaMemcpyAsync(ap.data(), h->d_ap[0] + R.cell_off + 1,
                              sizeof(unsigned long long) * m, cudaMemcpyDeviceToHost,
                              h->stream));
  CPM_CUDA(h, cudaMemcpyAsync(cs.data(), h->d_cs[0] + (R.cell_off + 1) * d,
                              sizeof(long long) * m * d, cudaMemcpyDeviceToHost, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  const int dims[3] = {R.nx, R.ny, R.nz};
  for (int c = 0; c < m; ++c)
    for (int k = 0; k < d; ++k) {
      double v = (double)cs[(size_t)c * d + k] / (double)unpack_area(ap[c]);
      if (std::isfinite(v)) v -= dims[k] * std::floor(v / dims[k]);
      out[(size_t)c * d + k] = v;
    }
  return CPM_OK;
}

int cpm_get_counters_r(cpm_handle* h, int r, cpm_counters* out) {
  if (!out || !h) return CPM_ERR_INVALID;
  if (r < -1 || r >= h->nrep)
    return h->fail(CPM_ERR_INVALID, "replica %d out of range", r);
  CPM_BIND(h);
  std::vector<unsigned long long> c(2 * h->nrep);
  CPM_CUDA(h, cudaMemcpyAsync(c.data(), h->d_counters, sizeof(unsigned long long) * 2 * h->nrep,
                              cudaMemcpyDeviceToHost, h->stream));
  CPM_CUDA(h, cudaStreamSynchronize(h->stream));
  out->attempts = out->evaluated = out->accepted = 0;
  for (int q = 0; q < h->nrep; ++q) {
    if (r >= 0 && q != r) continue;
    out->attempts += h->attempts[q];
    out->evaluated += c[2 * q];
    out->accepted += c[2 * q + 1];
  }
  return CPM_OK;
}

int cpm_get_counters(cpm_handle* h, cpm_counters* out) {
  return cpm_get_counters_r(h, -1, out);
}

int cpm_reset_counters(cpm_handle* h) {
  CPM_BIND(h);
  CPM_CUDA(h, cudaMemsetAsync(h->d_counters, 0, sizeof(unsigned long long) * 2 * h->nrep,
                              h->stream));
  std::fill(h->attempts.begin(), h->attempts.end(), 0ull);
  return CPM_OK;
}

int cpm_info(const cpm_handle* h, int* n_replicas, int* dimensionality,
             int* sweep_grid, uint64_t* kernel_launches) {
  if (!h) return CPM_ERR_INVALID;
  if (n_replicas) *n_replicas = h->nrep;
  if (dimensionality) *dimensionality = h->ndim;
  if (sweep_grid)
    *sweep_grid = uses_cluster(h) ? h->cluster_blocks : grid_of(h, run_variant(h), h->dispatch);
  if (kernel_launches) *kernel_launches = h->launches;
  return CPM_OK;
}

int cpm_sweep_config(const cpm_handle* h, int* variant, int* tile_x, int* tile_y,
                     int* tile_z, int* warps_per_block, int* grid, int* dispatch) {
  if (!h) return CPM_ERR_INVALID;
  if (variant) *variant = h->variant;
  const SweepPlan& p = plan_of(h, run_variant(h), h->dispatch);
  if (tile_x) *tile_x = 32;
  if (tile_y) *tile_y = p.rows;
  if (tile_z) *tile_z = 1;
  if (warps_per_block) *warps_per_block = p.warps;
  if (grid) *grid = p.grid;
  if (dispatch) *dispatch = h->dispatch;
  if (uses_cluster(h)) {  // one cluster, targets dealt one per lane
    if (tile_y) *tile_y = 1;
    if (warps_per_block) *warps_per_block = cluster_sweep_threads() / 32;
    if (grid) *grid = h->cluster_blocks;
  }
  return CPM_OK;
}

int cpm_debug_barrier_timeout(uint64_t timeout_ns, int* status) {
  if (!status) return CPM_ERR_INVALID;
  *status = 0;
  uint32_t* ctl = nullptr;
  cudaStream_t s = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&ctl, sizeof(uint32_t) * kCtlWords);
  if (e == cudaSuccess) e = cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * kCtlWords, s);
  if (e == cudaSuccess) e = launch_barrier_probe(ctl, timeout_ns, s);
  uint32_t w = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&w, ctl + kCtlErr, sizeof w, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(ctl);
  if (s) cudaStreamDestroy(s);
  if (e != cudaSuccess) {
    g_create_error = std::string("barrier probe failed: ") + cudaGetErrorString(e);
    return CPM_ERR_CUDA;
  }
  *status = (w & kErrTimeout) ? CPM_ERR_TIMEOUT : CPM_OK;
  return CPM_OK;
}

}  // extern "C"
