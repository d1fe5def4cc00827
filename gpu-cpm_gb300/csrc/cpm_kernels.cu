// cpm_kernels.cu — sm_103a kernels of the Cellular Potts engine around the
// sweep (cpm_sweep.cuh, cpm_cluster.cu).
//
//   init_pass1 / init_pass2    lattice validation and the table recount
//                              (area, perimeter, centroid sums).  Replaces
//                              calculateAreasAndCircumferences{,3d}
//                              (src/kernels2d.cu:5-41, src/kernels3d.cu:3-47).
//   init_prefdir_kernel, persist_fill_kernel, persist_update_kernel
//                              3D persistence: initial preferred directions,
//                              the mean-coordinate ring and the per-run
//                              direction update (src/kernels.cu:159-212).
//   lr_backward_kernel         likelihood-ratio gradient from score sums.
//   voronoi_kernel, voronoi_double_kernel
//                              periodic Voronoi seeding (bucketed, exact).
//   observe_heterotypic_kernel, observe_boundaries_kernel
//                              sorting order parameter and boundary lengths
//                              by type pair.
#include <algorithm>
#include <cstdint>

#include "cpm_device.cuh"
#include "cpm_sweep_common.cuh"

namespace gpucpm {
namespace {


__device__ __forceinline__ int find_site_replica(const DevReplica* reps,
                                                 int nrep, long long g) {
  int lo = 0, hi = nrep - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&reps[mid].lat_off) <= g)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}


// ---- table recount ---------------------------------------------------------

template <int NDIM>
__global__ void __launch_bounds__(kInitThreads)
    init_pass1(const uint32_t* __restrict__ lat,
               const DevReplica* __restrict__ reps, int nrep, long long total,
               unsigned long long* first, int* ctype, uint32_t* ctl) {
  int* err = reinterpret_cast<int*>(&ctl[kCtlErr]);
  const int lane = threadIdx.x & 31;
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
       g < total; g += (long long)gridDim.x * blockDim.x) {
    const int r = find_site_replica(reps, nrep, g);
    const long long local = g - __ldg(&reps[r].lat_off);
    const uint32_t v = lat[g];
    const uint32_t id = v & 0xFFFFFFu;
    const int ty = (int)(v >> 24);
    const bool bad = id > (uint32_t)__ldg(&reps[r].ncells);
    if (bad) atomicOr(err, kErrBadId);
    if (ty >= kMaxTypes) atomicOr(err, kErrBadType);
    if (id == 0 && ty != 0) atomicOr(err, kErrMediumType);
    const long long row = bad ? -1 : __ldg(&reps[r].cell_off) + id;
    // Lanes of one cell (neighbouring sites usually share one) check their
    // types against the lowest such lane, which holds the lowest site index
    // and alone updates the row.  Both words only change once in one
    // direction, so a row seen to be done already needs no atomic: of 2048^2
    // sites, 42,000 cells, most.
    const unsigned mask = __activemask();
    const unsigned peers = __match_any_sync(mask, (unsigned long long)row);
    const int leader = __ffs(peers) - 1;
    const int lty = __shfl_sync(mask, ty, leader);
    if (bad) continue;
    if (ty != lty) atomicOr(err, kErrTypeConflict);
    if (lane == leader) {
      if (__ldcg(&ctype[row]) != ty) {
        const int old = atomicCAS(&ctype[row], -1, ty);
        if (old != -1 && old != ty) atomicOr(err, kErrTypeConflict);
      }
      if (__ldcg(&first[row]) > (unsigned long long)local)
        atomicMin(&first[row], (unsigned long long)local);
    }
  }
}

// Every site of a cell adds 1 to its area, its number of foreign Moore
// neighbours to its perimeter, and its coordinates (periodic image nearest
// the cell's first site in raster order) to its centroid sums.
// Bound by its instructions: coordinates by reciprocals in 32 bits (64-bit
// divisions were most of them), and one set of additions per run of sites of
// a cell instead of one per site: recount of 2048^2 sites, 42,000 cells,
// 195 -> 161 us.
template <int NDIM>
__global__ void __launch_bounds__(kInitThreads)
    init_pass2(const uint32_t* __restrict__ lat,
               const DevReplica* __restrict__ reps, int nrep, long long total,
               const unsigned long long* __restrict__ first,
               unsigned long long* ap, long long* cs) {
  const int lane = threadIdx.x & 31;
  for (long long base = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; base < total;
       base += (long long)gridDim.x * blockDim.x) {  // (warp-uniform)
    const long long g = min(base + lane, total - 1);
    const DevReplica& R = reps[find_site_replica(reps, nrep, g)];
    const uint32_t v = lat[g];
    const uint32_t id = v & 0xFFFFFFu;
    const int nx = __ldg(&R.nx), ny = __ldg(&R.ny), nz = NDIM == 3 ? __ldg(&R.nz) : 1;
    const bool counts = base + lane < total && id != 0 && id <= (uint32_t)__ldg(&R.ncells);
    const long long row = counts ? __ldg(&R.cell_off) + id : -1;
    const int dim[3] = {nx, ny, nz};
    int foreign = 0, image[3] = {0, 0, 0};
    if (counts) {
      const long long off = __ldg(&R.lat_off);
      const FastDiv div_nx = {__ldg(&R.div_nx.mul), __ldg(&R.div_nx.shift)},
                    div_plane = {__ldg(&R.div_plane.mul), __ldg(&R.div_plane.shift)};
      const unsigned plane = (unsigned)nx * (unsigned)ny;
      auto coords = [&](const unsigned site, int (&c)[3]) {
        c[2] = NDIM == 3 ? (int)fast_div(site, div_plane) : 0;
        const unsigned in_plane = site - (unsigned)c[2] * plane;
        c[1] = (int)fast_div(in_plane, div_nx);
        c[0] = (int)(in_plane - (unsigned)c[1] * (unsigned)nx);
      };
      int c[3], anchor[3];
      coords((unsigned)(g - off), c);
      coords((unsigned)first[row], anchor);
      const uint32_t* L = lat + off;
#pragma unroll
      for (int dz = (NDIM == 3 ? -1 : 0); dz <= (NDIM == 3 ? 1 : 0); ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
          for (int dx = -1; dx <= 1; ++dx) {
            if (!dz && !dy && !dx) continue;
            const unsigned zz = (unsigned)wrap_coord(c[2] + dz, nz),
                           yy = (unsigned)wrap_coord(c[1] + dy, ny),
                           xx = (unsigned)wrap_coord(c[0] + dx, nx);
            foreign += L[(NDIM == 3 ? zz * plane : 0u) + yy * (unsigned)nx + xx] != v;
          }
#pragma unroll
      for (int k = 0; k < NDIM; ++k) {
        const long long d = 2LL * (c[k] - anchor[k]);
        image[k] = d > dim[k] ? c[k] - dim[k] : (d < -dim[k] ? c[k] + dim[k] : c[k]);
      }
    }
    // Sums over each run of lanes of one cell, added by its last lane (sums of
    // 32 coordinates in 32 bits; where sides are too long for that every lane
    // is a run).
    const bool fits = max(nx, max(ny, nz)) < (1 << 24);
    const long long before = __shfl_up_sync(kFull, row, 1);
    const unsigned heads = __ballot_sync(kFull, lane == 0 || row != before || !fits);
    const int head = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int f = __shfl_up_sync(kFull, foreign, o);
      int u[NDIM];
#pragma unroll
      for (int k = 0; k < NDIM; ++k) u[k] = __shfl_up_sync(kFull, image[k], o);
      if (lane - o >= head) {
        foreign += f;
#pragma unroll
        for (int k = 0; k < NDIM; ++k) image[k] += u[k];
      }
    }
    if (counts && (lane == 31 || (heads >> (lane + 1)) & 1u)) {
      atomicAdd(ap + row, pack_delta(lane - head + 1, foreign));
#pragma unroll
      for (int k = 0; k < NDIM; ++k)
        atomicAdd(reinterpret_cast<unsigned long long*>(&cs[row * NDIM + k]),
                  (unsigned long long)(long long)image[k]);
    }
  }
}

// Failure-detection probe: every block waits at a barrier episode that
// needs twice the blocks the grid has, so the bounded wait runs out and the
// error word records kErrTimeout.  No memory beyond ctl[] is touched.
__global__ void barrier_probe(uint32_t* ctl, unsigned long long timeout_ns) {
  __shared__ int s_ok;
  grid_barrier(ctl, 2u, &s_ok, timeout_ns);
}

// ---- likelihood-ratio backward ---------------------------------------------
struct Checkpoints {
  int n;
  int t[kMaxCheckpoints];
  // Baseline over replicas beyond this launch's (replicas sharded over
  // processes): sum of O[.][c] and replica count of all shards.
  int use_total;
  int nrep_total;
  float total[kMaxCheckpoints];
};

// grad[k] = sum_r sum_c dL/dO[r][c] (O[r][c] - b[r][c])
//                     * sum_{t < checkpoints[c]} scores[r][t][k]
// with the leave-one-out baseline b[r][c] = mean of O[.][c] over the other
// replicas (0 for a single replica), so that each replica's term is an
// unbiased estimate of dE[O]/dtheta scaled by dL/dO[r][c].  With use_total
// the other replicas are those of every shard (total / nrep_total).
// One block per parameter k; threads stride over replicas, each walking its
// replica's scores once in time order while passing the checkpoints.
__global__ void lr_backward_kernel(const float* __restrict__ scores,
                                   const float* __restrict__ dl_do,
                                   const float* __restrict__ obs, const Checkpoints cp,
                                   int nrep, int len, float* grad) {
  const int ncheck = cp.n;
  const int k = blockIdx.x;
  __shared__ float s_mean[kMaxCheckpoints];  // sum over replicas
  __shared__ float s_red[32];
  for (int c = threadIdx.x; c < ncheck; c += blockDim.x) {
    float m = 0.0f;
    if (cp.use_total) {
      m = cp.total[c];
    } else {
      for (int r = 0; r < nrep; ++r) m += obs[(long long)r * ncheck + c];
    }
    s_mean[c] = m;
  }
  const int nall = cp.use_total ? cp.nrep_total : nrep;
  __syncthreads();
  float acc = 0.0f;
  for (int r = threadIdx.x; r < nrep; r += blockDim.x) {
    float cum = 0.0f;
    int t = 0;
    for (int c = 0; c < ncheck; ++c) {
      const int upto = min(cp.t[c], len);
      for (; t < upto; ++t) cum += scores[((long long)r * len + t) * kScoreMax + k];
      const long long rc = (long long)r * ncheck + c;
      const float o = obs[rc];
      const float dev = nall > 1 ? o - (s_mean[c] - o) / (float)(nall - 1) : o;
      acc += dl_do[rc] * dev * cum;
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (int)(blockDim.x >> 5) ? s_red[threadIdx.x] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (threadIdx.x == 0) grad[k] = v;
  }
}

// ---- 3D persistence ----------------------------------------------------------
__device__ __forceinline__ int find_row_replica(const DevReplica* reps, int nrep, long long row) {
  int lo = 0, hi = nrep - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&reps[mid].cell_off) <= row)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Initial preferred directions: uniform on the sphere, by rejection from the
// cube [-1, 1)^3 with Philox draws of counter (cell, 0xFFFFFFF0 - try,
// stream, 0xFFFFFFFF) (outside the sweep's phases), normalised in double.
// The reference draws normalised Gaussians from std::random_device
// (src/cpm.cu:226-248).
__global__ void init_prefdir_kernel(double* prefdir, const DevReplica* __restrict__ reps,
                                    int nrep, long long rows, unsigned long long seed,
                                    unsigned stream0) {
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
       row += (long long)gridDim.x * blockDim.x) {
    const int r = find_row_replica(reps, nrep, row);
    const uint32_t cell = (uint32_t)(row - __ldg(&reps[r].cell_off));
    double d[3] = {1.0, 0.0, 0.0};
    for (uint32_t tr = 0; tr < 64; ++tr) {
      uint32_t c0 = cell, c1 = 0xFFFFFFF0u - tr, c2 = stream0 + (uint32_t)r, c3 = 0xFFFFFFFFu;
      philox4x32_10(c0, c1, c2, c3, k0, k1);
      const double x = (double)(c0 >> 8) * 0x1p-23 - 1.0;
      const double y = (double)(c1 >> 8) * 0x1p-23 - 1.0;
      const double z = (double)(c2 >> 8) * 0x1p-23 - 1.0;
      const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
      if (r2 > 0.0 && r2 <= 1.0) {
        const double l = __dsqrt_rn(r2);
        d[0] = __ddiv_rn(x, l);
        d[1] = __ddiv_rn(y, l);
        d[2] = __ddiv_rn(z, l);
        break;
      }
    }
    prefdir[3 * row + 0] = d[0];
    prefdir[3 * row + 1] = d[1];
    prefdir[3 * row + 2] = d[2];
  }
}

// Mean coordinate of a cell on one axis, in [0, n): exact sum / area.
__device__ __forceinline__ double mean_coord(long long sum, long long area, int n) {
  double m = __ddiv_rn((double)sum, (double)area);
  m = __dsub_rn(m, __dmul_rn((double)n, floor(__ddiv_rn(m, (double)n))));
  return m;
}

// hist slots [H][rows][3] all set to the cells' current mean coordinates
// (the reference fills its history at every push, src/cpm.cu:578-583).
__global__ void persist_fill_kernel(double* hist, int H, const unsigned long long* __restrict__ ap,
                                    const long long* __restrict__ cs,
                                    const DevReplica* __restrict__ reps, int nrep, long long rows) {
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
       row += (long long)gridDim.x * blockDim.x) {
    const int r = find_row_replica(reps, nrep, row);
    const long long area = unpack_area(__ldg(ap + row));
    const int dims[3] = {__ldg(&reps[r].nx), __ldg(&reps[r].ny), __ldg(&reps[r].nz)};
    for (int k = 0; k < 3; ++k) {
      const double m = area > 0 ? mean_coord(__ldg(cs + 3 * row + k), area, dims[k]) : 0.0;
      for (int h = 0; h < H; ++h) hist[((long long)h * rows + row) * 3 + k] = m;
    }
  }
}

// After a run: the current mean goes into history slot `slot`; the mean of
// slot (slot + 1) % H (H runs ago, the oldest) gives the displacement d.
// As src/kernels.cu:159-212: d is divided by its length taken before the
// per-axis wrap into (-n/2, n/2], then the preferred direction becomes
// normalize(d (1 - p) + pref p) with p the cell type's diffusion; cells with
// no displacement (or no sites) keep theirs.  Double precision throughout.
__global__ void persist_update_kernel(double* prefdir, double* hist, int H, int slot,
                                      const unsigned long long* __restrict__ ap,
                                      const long long* __restrict__ cs,
                                      const int* __restrict__ ctype,
                                      const DevParams* __restrict__ params,
                                      const DevReplica* __restrict__ reps, int nrep,
                                      long long rows) {
  for (long long row = (long long)blockIdx.x * blockDim.x + threadIdx.x; row < rows;
       row += (long long)gridDim.x * blockDim.x) {
    const int r = find_row_replica(reps, nrep, row);
    const long long cell = row - __ldg(&reps[r].cell_off);
    const long long area = unpack_area(__ldg(ap + row));
    const int dims[3] = {__ldg(&reps[r].nx), __ldg(&reps[r].ny), __ldg(&reps[r].nz)};
    double cur[3], d[3];
    for (int k = 0; k < 3; ++k) {
      cur[k] = area > 0 ? mean_coord(__ldg(cs + 3 * row + k), area, dims[k]) : 0.0;
      hist[((long long)slot * rows + row) * 3 + k] = cur[k];
    }
    const int prev_slot = (slot + 1) % H;
    for (int k = 0; k < 3; ++k)
      d[k] = __dsub_rn(cur[k], hist[((long long)prev_slot * rows + row) * 3 + k]);
    if (cell == 0 || area <= 0) continue;
    const double len = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])),
                                            __dmul_rn(d[2], d[2])));
    if (len == 0.0) continue;
    const int ty = __ldg(ctype + row);
    if (ty < 0 || ty >= kMaxTypes) continue;
    const double p = (double)__ldg(&params[__ldg(&reps[r].pset)].persist_diff[ty]);
    double np[3];
    for (int k = 0; k < 3; ++k) {
      double v = d[k];
      if (v > (double)(dims[k] / 2)) v = __dsub_rn(v, (double)dims[k]);
      if (v < (double)(-(dims[k] / 2))) v = __dadd_rn(v, (double)dims[k]);
      v = __ddiv_rn(v, len);
      np[k] = __dadd_rn(__dmul_rn(v, __dsub_rn(1.0, p)), __dmul_rn(prefdir[3 * row + k], p));
    }
    const double l2 = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(np[0], np[0]), __dmul_rn(np[1], np[1])),
                                           __dmul_rn(np[2], np[2])));
    if (l2 == 0.0) continue;
    for (int k = 0; k < 3; ++k) prefdir[3 * row + k] = __ddiv_rn(np[k], l2);
  }
}

// ---- sorting order parameter -------------------------------------------------
// Per replica: number of Moore neighbour pairs (each pair once) of two
// different non-medium cells, and how many of them join cells of different
// types.  counts[2 r] = all such pairs, counts[2 r + 1] = heterotypic ones.
//
// A warp takes tasks of 32 columns x kObserveRows rows of one replica (`start`:
// tasks before each replica): a lane walks its column, so the row below's
// three loads are the next row's centre and right neighbour.  Bound: reading
// the lattice.  Counts stay in registers from task to task, then in shared
// memory for the block's first replica (its tasks are one contiguous run),
// so a block issues two global atomics per replica it meets.  (One 64-bit
// atomic pair per counted site, on two addresses per replica, took 1.18 ms on
// a 2048^2 tissue and ~10 ms on 256 replicas of 45.5 M sites together.)
__global__ void __launch_bounds__(256)
    observe_heterotypic_kernel(const uint32_t* __restrict__ lat,
                               const DevReplica* __restrict__ reps, int nrep,
                               const long long* __restrict__ start,
                               unsigned long long* counts) {
  __shared__ unsigned long long s_sum[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0ull;
  __syncthreads();
  const long long ntasks = __ldg(start + nrep);
  const long long per = (ntasks + gridDim.x - 1) / gridDim.x;
  const long long t0 = (long long)blockIdx.x * per, t1 = min(ntasks, t0 + per);
  auto find = [&](long long t, int lo) {  // the replica of task t, at or after lo
    int hi = nrep - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(start + mid) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
  };
  const int rep0 = t0 < t1 ? find(t0, 0) : 0;
  int r = rep0;
  unsigned long long pairs = 0, hetero = 0;  // this lane's counts of replica r
  auto flush = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      pairs += __shfl_xor_sync(kFull, pairs, o);
      hetero += __shfl_xor_sync(kFull, hetero, o);
    }
    if (lane == 0 && pairs) {
      unsigned long long* dst = r == rep0 ? s_sum : counts + 2LL * r;
      atomicAdd(dst, pairs);
      if (hetero) atomicAdd(dst + 1, hetero);
    }
    pairs = hetero = 0;
  };
  for (long long t = t0 + warp; t < t1; t += wpb) {
    if (t >= __ldg(start + r + 1)) {
      flush();
      r = find(t, r);
    }
    const int nx = __ldg(&reps[r].nx), ny = __ldg(&reps[r].ny);
    const uint32_t* L = lat + __ldg(&reps[r].lat_off);
    const int local = (int)(t - __ldg(start + r)), segs = (nx + 31) >> 5;
    const int x = (local % segs) * 32 + lane, y0 = (local / segs) * kObserveRows;
    const int rows = min(kObserveRows, ny - y0);
    if (x >= nx) continue;
    const int xl = x ? x - 1 : nx - 1, xr = x + 1 < nx ? x + 1 : 0;
    const uint32_t* row = L + (long long)y0 * nx;
    uint32_t v = __ldg(row + x), right = __ldg(row + xr);
    unsigned np = 0, nh = 0;
    auto pair = [&](uint32_t w) {
      const bool p = (v & 0xFFFFFFu) && (w & 0xFFFFFFu) && w != v;
      np += p;
      nh += p && (w >> 24) != (v >> 24);
    };
#pragma unroll 4
    for (int k = 0; k < rows; ++k) {
      // forward half of the Moore neighbourhood: (0,1), (1,-1), (1,0), (1,1)
      row = y0 + k + 1 < ny ? row + nx : L;
      const uint32_t l = __ldg(row + xl), c = __ldg(row + x), rr = __ldg(row + xr);
      pair(right);
      pair(l);
      pair(c);
      pair(rr);
      v = c;
      right = rr;
    }
    pairs += np;
    hetero += nh;
  }
  __syncwarp();
  flush();
  __syncthreads();
  if (threadIdx.x < 2 && s_sum[threadIdx.x])
    atomicAdd(counts + 2LL * rep0 + threadIdx.x, s_sum[threadIdx.x]);
}

// ---- periodic Voronoi seeding -------------------------------------------------
// One thread per site.  Buckets are scanned ring by ring (Chebyshev distance
// r in bucket units, wrapped; a bucket met twice through the wrap changes
// nothing) until the best squared distance is below the squared lower bound
// r * min(w) of every bucket not yet scanned, so the answer is the exact
// brute-force nearest point with ties to the lowest index.
//
// The rings are scanned in FP32 first, keeping the nearest point and the
// distance of the second nearest: this chip has 2 FP64 lanes per SM, and a
// distance takes 11 FP64 operations (2048^2 sites, 42,000 points: 5.96 ms all
// in FP64).  A float distance is off by at most vg.ferr, so a nearest point
// that leads by more than 2 ferr is the answer; only where the lead is
// smaller (ties, points midway) are the site's rings scanned in double.  On
// lattices so long that ferr is no longer small against a bucket
// (VoronoiGrid::single) voronoi_double_kernel scans them in double alone.
__device__ __forceinline__ double min_image(double a, double b, int n) {
  const double d = fabs(__dsub_rn(a, b));
  const double e = __dsub_rn((double)n, d);
  return e < d ? e : d;
}

// Bucket coordinate b of an axis of g buckets, wrapped.
__device__ __forceinline__ int wrap_bucket(int b, int g) {
  if (b < 0) b += g;
  if (b >= g) b -= g;
  if (b < 0 || b >= g) {  // (rings wider than this axis)
    b %= g;
    b += b < 0 ? g : 0;
  }
  return b;
}

// visit(k0, k1) for the points of every bucket of ring r around bucket b.
template <int NDIM, class F>
__device__ __forceinline__ void scan_ring(const VoronoiGrid& vg, const int* __restrict__ start,
                                          const int (&b)[3], int r, F&& visit) {
  const int zr = NDIM == 3 ? r : 0;
  for (int dz = -zr; dz <= zr; ++dz) {
    const int bz = NDIM == 3 ? wrap_bucket(b[2] + dz, vg.g[2]) : 0;
    for (int dy = -r; dy <= r; ++dy) {
      const int row = (bz * vg.g[1] + wrap_bucket(b[1] + dy, vg.g[1])) * vg.g[0];
      // the shell of ring r: whole rows on its faces, else the two ends
      const bool face = dy == r || dy == -r || (NDIM == 3 && (dz == r || dz == -r));
      for (int dx = -r; dx <= r; dx += face || r == 0 ? 1 : 2 * r) {
        const int bucket = row + wrap_bucket(b[0] + dx, vg.g[0]);
        visit(__ldg(start + bucket), __ldg(start + bucket + 1));
      }
    }
  }
}

// The nearest point so far, in double, ties to the lowest index.
struct Nearest {
  double d2 = 1e300;
  int k = 0x7FFFFFFF;
};
template <int NDIM>
__device__ __forceinline__ void take_nearer(const VoronoiGrid& vg, const double* __restrict__ pts,
                                            const int* __restrict__ idx, int j, int x, int y,
                                            int z, Nearest& best) {
  const double ddx = min_image((double)x, __ldg(pts + 3LL * j), vg.n[0]);
  const double ddy = min_image((double)y, __ldg(pts + 3LL * j + 1), vg.n[1]);
  double d2 = __dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy));
  if (NDIM == 3) {
    const double ddz = min_image((double)z, __ldg(pts + 3LL * j + 2), vg.n[2]);
    d2 = __dadd_rn(d2, __dmul_rn(ddz, ddz));
  }
  const int k = __ldg(idx + j);
  if (d2 < best.d2 || (d2 == best.d2 && k < best.k)) {
    best.d2 = d2;
    best.k = k;
  }
}

// The points in bucket order, in FP64 and FP32: point idx[j] at place j.  A few
// microseconds of latency.
__global__ void __launch_bounds__(256)
    voronoi_order_kernel(int ndim, int npoints, const double* __restrict__ raw,
                         const int* __restrict__ idx, double* pts, float4* fpts) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npoints) return;
  const double* p = raw + (long long)__ldg(idx + j) * ndim;
  const double x = __ldg(p), y = __ldg(p + 1), z = ndim == 3 ? __ldg(p + 2) : 0.0;
  double* q = pts + 3LL * j;
  q[0] = x, q[1] = y, q[2] = z;
  fpts[j] = make_float4((float)x, (float)y, (float)z, 0.0f);
}

template <int NDIM>
__global__ void __launch_bounds__(256)
    voronoi_kernel(uint32_t* lat, const VoronoiGrid vg, const double* __restrict__ pts,
                   const float4* __restrict__ fpts, const int* __restrict__ idx,
                   const uint32_t* __restrict__ values, const int* __restrict__ start) {
  const unsigned sites = (unsigned)vg.n[0] * vg.n[1] * vg.n[2];  // < 2^31
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < sites;
       s += gridDim.x * blockDim.x) {
    const int x = (int)(s % vg.n[0]), yz = (int)(s / vg.n[0]);
    const int y = NDIM == 3 ? yz % vg.n[1] : yz, z = NDIM == 3 ? yz / vg.n[1] : 0;
    const int xyz[3] = {x, y, z};
    int b[3];
    float edge = 3.0e38f;  // distance to the nearest edge of the site's bucket
#pragma unroll
    for (int a = 0; a < NDIM; ++a) {  // (FP32: ferr covers a bucket off at its edge)
      const float c = (float)xyz[a];
      b[a] = (int)floorf(c * vg.inv_w[a]);
      b[a] = min(max(b[a], 0), vg.g[a] - 1);
      const float lo = c - (float)b[a] * vg.wf[a];
      edge = fminf(edge, fminf(lo, vg.wf[a] - lo));
    }
    if (NDIM == 2) b[2] = 0;
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    const float nx = (float)vg.n[0], ny = (float)vg.n[1], nz = (float)vg.n[2];
    auto dist2 = [&](const float4 p) {
      float dx = fabsf(fx - p.x), dy = fabsf(fy - p.y);
      dx = fminf(dx, nx - dx);
      dy = fminf(dy, ny - dy);
      float d2 = dx * dx + dy * dy;
      if (NDIM == 3) {
        float dz = fabsf(fz - p.z);
        dz = fminf(dz, nz - dz);
        d2 = d2 + dz * dz;
      }
      return d2;
    };
    float best = 3.0e38f, second = 3.0e38f;  // squared, of two different points
    int best_j = -1;                         // position in bucket order
    int r = 0;
    for (; r <= vg.rmax; ++r) {
      scan_ring<NDIM>(vg, start, b, r, [&](int k0, int k1) {
        for (int k = k0; k < k1; ++k) {
          const float d2 = dist2(__ldg(fpts + k));
          if (k == best_j) continue;
          second = fminf(second, fmaxf(best, d2));
          if (d2 < best) {
            best = d2;
            best_j = k;
          }
        }
      });
      // every bucket not scanned yet lies at periodic Chebyshev distance
      // >= r + 1, so its points are at least r * min(w) + edge away
      const float lb = (float)r * vg.lb_scale + edge - 3.0f * vg.ferr;
      if (best_j >= 0 && lb > 0.0f && best < lb * lb) break;
    }
    const float lead = sqrtf(best) + 2.0f * vg.ferr, lead2 = lead * lead;
    uint32_t out = 0;
    if (best_j >= 0 && second > lead2) {
      out = __ldg(values + __ldg(idx + best_j));
    } else {  // the points that may be nearest, in double
      Nearest near;
      for (int q = 0; q <= min(r, vg.rmax); ++q) {
        scan_ring<NDIM>(vg, start, b, q, [&](int k0, int k1) {
          for (int k = k0; k < k1; ++k)
            if (dist2(__ldg(fpts + k)) <= lead2)
              take_nearer<NDIM>(vg, pts, idx, k, x, y, z, near);
        });
      }
      if (near.k != 0x7FFFFFFF) out = __ldg(values + near.k);
    }
    lat[s] = out;
  }
}

// The same in double alone.
template <int NDIM>
__global__ void __launch_bounds__(256)
    voronoi_double_kernel(uint32_t* lat, const VoronoiGrid vg, const double* __restrict__ pts,
                          const int* __restrict__ idx, const uint32_t* __restrict__ values,
                          const int* __restrict__ start) {
  const unsigned sites = (unsigned)vg.n[0] * vg.n[1] * vg.n[2];  // < 2^31
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < sites;
       s += gridDim.x * blockDim.x) {
    const int x = (int)(s % vg.n[0]), yz = (int)(s / vg.n[0]);
    const int y = NDIM == 3 ? yz % vg.n[1] : yz, z = NDIM == 3 ? yz / vg.n[1] : 0;
    const int xyz[3] = {x, y, z};
    int b[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < NDIM; ++a)
      b[a] = min((int)__dmul_rn((double)xyz[a], vg.inv[a]), vg.g[a] - 1);
    Nearest near;
    for (int r = 0; r <= vg.rmax; ++r) {
      scan_ring<NDIM>(vg, start, b, r, [&](int k0, int k1) {
        for (int k = k0; k < k1; ++k) take_nearer<NDIM>(vg, pts, idx, k, x, y, z, near);
      });
      // every bucket not scanned yet lies r * wmin away at least; the margin
      // covers the rounding of the bucket indices
      const double lb = __dsub_rn(__dmul_rn((double)r, vg.wmin), 1e-6);
      if (near.k != 0x7FFFFFFF && lb > 0.0 && near.d2 < __dmul_rn(lb, lb)) break;
    }
    lat[s] = near.k != 0x7FFFFFFF ? __ldg(values + near.k) : 0u;
  }
}

// ---- boundary counts per type pair ------------------------------------------
// A block takes tiles of kBoundaryTile sites of one replica, histograms the
// pairs in shared memory and adds the non-zero bins to global memory.
template <int NDIM>
__global__ void observe_boundaries_kernel(const uint32_t* __restrict__ lat,
                                          const DevReplica* __restrict__ reps, int nrep,
                                          const long long* __restrict__ tile_start,
                                          long long ntiles, int T,
                                          unsigned long long* counts) {
  extern __shared__ unsigned int hist[];  // T * T
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int lo = 0, hi = nrep - 1;  // the replica owning tile t
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(tile_start + mid) <= t) lo = mid; else hi = mid - 1;
    }
    const int r = lo;
    const DevReplica R = reps[r];
    const long long sites = (long long)R.nx * R.ny * R.nz;
    const long long first = (t - __ldg(tile_start + r)) * kBoundaryTile;
    for (int i = threadIdx.x; i < T * T; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (long long local = first + threadIdx.x;
         local < sites && local < first + kBoundaryTile; local += blockDim.x) {
      const int x = (int)(local % R.nx), y = (int)((local / R.nx) % R.ny),
                z = (int)(local / ((long long)R.nx * R.ny));
      const uint32_t v = lat[R.lat_off + local];
      const int tv = (int)(v >> 24);
      // forward half of the neighbourhood: offsets after (0,0,0) in
      // (dz, dy, dx) row-major order
      for (int m = (NDIM == 3 ? 14 : 5); m < (NDIM == 3 ? 27 : 9); ++m) {
        const int ox = m % 3 - 1, oy = (m / 3) % 3 - 1, oz = NDIM == 3 ? m / 9 - 1 : 0;
        int xx = x + ox, yy = y + oy, zz = z + oz;
        xx = xx < 0 ? xx + R.nx : (xx >= R.nx ? xx - R.nx : xx);
        yy = yy < 0 ? yy + R.ny : (yy >= R.ny ? yy - R.ny : yy);
        zz = zz < 0 ? zz + R.nz : (zz >= R.nz ? zz - R.nz : zz);
        const uint32_t w = lat[R.lat_off + ((long long)zz * R.ny + yy) * R.nx + xx];
        if (w == v) continue;
        const int tw = (int)(w >> 24);
        if (tv >= T || tw >= T) continue;
        const int a = tv < tw ? tv : tw, bb = tv < tw ? tw : tv;
        atomicAdd(&hist[a * T + bb], 1u);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T * T; i += blockDim.x)
      if (hist[i]) atomicAdd(&counts[(long long)r * T * T + i], (unsigned long long)hist[i]);
    __syncthreads();
  }
}

}  // namespace

cudaError_t launch_voronoi(uint32_t* lat, const VoronoiGrid& vg, int npoints, const double* raw,
                           double* pts, float4* fpts, const int* idx, const uint32_t* values,
                           const int* start, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long sites = (long long)vg.n[0] * vg.n[1] * vg.n[2];
  const int grid = (int)std::max(1LL, std::min<long long>((sites + 255) / 256, (long long)sms * 16));
  voronoi_order_kernel<<<(npoints + 255) / 256, 256, 0, s>>>(vg.ndim, npoints, raw, idx, pts,
                                                             fpts);
  if (!vg.single) {
    if (vg.ndim == 2)
      voronoi_double_kernel<2><<<grid, 256, 0, s>>>(lat, vg, pts, idx, values, start);
    else
      voronoi_double_kernel<3><<<grid, 256, 0, s>>>(lat, vg, pts, idx, values, start);
  } else if (vg.ndim == 2)
    voronoi_kernel<2><<<grid, 256, 0, s>>>(lat, vg, pts, fpts, idx, values, start);
  else
    voronoi_kernel<3><<<grid, 256, 0, s>>>(lat, vg, pts, fpts, idx, values, start);
  return cudaGetLastError();
}

cudaError_t launch_observe_boundaries(int ndim, const uint32_t* lat, const DevReplica* reps,
                                      int nrep, const long long* tile_start, long long ntiles,
                                      int T, unsigned long long* counts, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)std::max(1LL, std::min<long long>(ntiles, (long long)sms * 8));
  const size_t shm = sizeof(unsigned int) * T * T;
  if (ndim == 2)
    observe_boundaries_kernel<2><<<grid, 256, shm, s>>>(lat, reps, nrep, tile_start, ntiles, T,
                                                        counts);
  else
    observe_boundaries_kernel<3><<<grid, 256, shm, s>>>(lat, reps, nrep, tile_start, ntiles, T,
                                                        counts);
  return cudaGetLastError();
}

cudaError_t launch_lr_backward(const float* scores, const float* dl_do,
                               const float* obs, const int* checkpoints, int nrep,
                               int len, int nparam, int ncheck, const float* obs_total,
                               int nrep_total, float* grad, cudaStream_t s) {
  if (ncheck < 1 || ncheck > kMaxCheckpoints || nparam < 1 || nparam > kScoreMax)
    return cudaErrorInvalidValue;
  Checkpoints cp;
  cp.n = ncheck;
  cp.use_total = obs_total ? 1 : 0;
  cp.nrep_total = nrep_total;
  for (int c = 0; c < ncheck; ++c) {
    cp.t[c] = checkpoints[c];
    cp.total[c] = obs_total ? obs_total[c] : 0.0f;
  }
  lr_backward_kernel<<<nparam, 256, 0, s>>>(scores, dl_do, obs, cp, nrep, len, grad);
  return cudaGetLastError();
}

namespace {
int rows_grid(long long rows) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long want = (rows + 255) / 256;
  return (int)std::max(1LL, std::min<long long>(want, (long long)sms * 8));
}
}  // namespace

cudaError_t launch_init_prefdir(double* prefdir, const DevReplica* reps, int nrep,
                                long long rows, unsigned long long seed, unsigned stream0,
                                cudaStream_t s) {
  init_prefdir_kernel<<<rows_grid(rows), 256, 0, s>>>(prefdir, reps, nrep, rows, seed, stream0);
  return cudaGetLastError();
}

cudaError_t launch_persist_fill(double* hist, int H, const unsigned long long* ap,
                                const long long* cs, const DevReplica* reps, int nrep,
                                long long rows, cudaStream_t s) {
  persist_fill_kernel<<<rows_grid(rows), 256, 0, s>>>(hist, H, ap, cs, reps, nrep, rows);
  return cudaGetLastError();
}

cudaError_t launch_persist_update(double* prefdir, double* hist, int H, int slot,
                                  const unsigned long long* ap, const long long* cs,
                                  const int* ctype, const DevParams* params,
                                  const DevReplica* reps, int nrep, long long rows,
                                  cudaStream_t s) {
  persist_update_kernel<<<rows_grid(rows), 256, 0, s>>>(prefdir, hist, H, slot, ap, cs, ctype,
                                                        params, reps, nrep, rows);
  return cudaGetLastError();
}

cudaError_t launch_observe_heterotypic(const uint32_t* lat, const DevReplica* reps,
                                       int nrep, const long long* start, long long ntasks,
                                       unsigned long long* counts, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid =
      (int)std::max(1LL, std::min<long long>((ntasks + 7) / 8, (long long)sms * 8));
  observe_heterotypic_kernel<<<grid, 256, 0, s>>>(lat, reps, nrep, start, counts);
  return cudaGetLastError();
}

cudaError_t launch_barrier_probe(uint32_t* ctl, unsigned long long timeout_ns,
                                 cudaStream_t s) {
  void* args[] = {&ctl, &timeout_ns};
  return cudaLaunchCooperativeKernel((const void*)barrier_probe, dim3(2), dim3(32),
                                     args, 0, s);
}

cudaError_t launch_init(int ndim, const uint32_t* lat, const DevReplica* reps,
                        int nrep, long long total_sites, unsigned long long* ap,
                        long long* cs, unsigned long long* first, int* ctype,
                        uint32_t* ctl, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long want = (total_sites + kInitThreads - 1) / kInitThreads;
  const int grid = (int)(want < (long long)sms * 8 ? (want > 0 ? want : 1)
                                                   : (long long)sms * 8);
  if (ndim == 2) {
    init_pass1<2><<<grid, kInitThreads, 0, s>>>(lat, reps, nrep, total_sites,
                                                 first, ctype, ctl);
    init_pass2<2><<<grid, kInitThreads, 0, s>>>(lat, reps, nrep, total_sites,
                                                 first, ap, cs);
  } else {
    init_pass1<3><<<grid, kInitThreads, 0, s>>>(lat, reps, nrep, total_sites,
                                                 first, ctype, ctl);
    init_pass2<3><<<grid, kInitThreads, 0, s>>>(lat, reps, nrep, total_sites,
                                                 first, ap, cs);
  }
  return cudaGetLastError();
}

}  // namespace gpucpm
