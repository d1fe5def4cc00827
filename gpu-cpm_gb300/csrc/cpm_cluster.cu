// cpm_cluster.cu — the sweep of a small single 2D lattice by one thread-block
// cluster.
//
//   cluster_sweep_kernel  the checkerboard Metropolis sweep (cpm_sweep.cuh:
//                         same schedule, random stream and FP32 operation
//                         order, so its results are bit-identical) of one 2D
//                         lattice that fits the shared memory of a cluster,
//                         tables included.  Replaces copyAttempt
//                         (src/kernels2d.cu:44-583) for these lattices.
//
// A phase of a small lattice is all latency: the grid sweep's takes 4.6 us at
// 256^2, of which the grid barrier is 1.5 and the L2 round trips of sites,
// table rows and replayed deltas most of the rest.  Here nothing leaves the
// cluster between the first load and the last store:
//  * Block k keeps lattice rows [k H, k H + H) with one halo row above and one
//    below (copies of the neighbouring blocks' edge rows) and a periodic
//    column on each side.  Targets lie in the block's own rows; a write to an
//    edge row also goes into the neighbour's halo, to an edge column into its
//    copy.  A halo row is read only in phases that write rows of other
//    classes.
//  * Every block keeps the whole area / perimeter / centroid tables.  A row
//    that a copy changes is an 8-byte message in the block's outbox; at the
//    start of the next phase warp w of every block reads block w's outbox
//    (distributed shared memory), its loads in flight over the phase's queueing,
//    and applies it to the block's tables.  So tables are as they stood when
//    the phase began when its attempts read them, without a second copy or a
//    replay.  Where whole tables do not fit, their rows are dealt over the
//    blocks (DEALT), changed by their owner and read from it, which needs a
//    second cluster barrier per phase: 256^2 of 6,000 rows, 50 MCS 743 us, of
//    5,000 in whole tables 568.
//  * Phases end at the cluster's hardware barrier (509 cycles; with the tables
//    in global memory it waited for the reductions too, 2,019).
// The block's attempts are queued together and evaluated on two lanes each
// (pair_energy): a phase is one warp's chain through one batch of them.
// The next phase's draws, which need neither sites nor tables, are made
// between arriving at the barrier and waiting for it.
//
// Bound: one warp's chain (256^2, cycles of 5,400: queueing 1,050, messages and
// block barrier 1,000, one batch of attempts 2,350, cluster barrier 950).
// Measured, 1000 MCS on the 256^2 sorting lattice: grid sweep 18.5 ms, the
// cluster sweep before this one (tables in global memory, a warp tile at a
// time) 14.4 ms, this one 10.9 ms; 10 MCS and a pull of the 200^2 lattice 221
// -> 143 us.  By size (us per MCS, grid / cluster): 64^2 17.0 / 9.0, 256^2 18.9 /
// 10.1, 350^2 19.5 / 16.7, 400^2 19.2 / 20.4.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>

#include "cpm_device.cuh"
#include "cpm_sweep_common.cuh"

namespace gpucpm {
namespace {

// 512 threads, two targets of a lane side by side: 1000 MCS at 256^2 10.9 ms
// (one target 11.6; before the draws moved behind the barrier's arrival 256
// threads with four targets took 13.3, 128 with eight 20.0 against 11.6).
constexpr int kClusterThreads = 512;
constexpr int kRoundTargets = 2;
constexpr int kSources = 16 / (kClusterThreads / 32);  // blocks whose messages a warp reads

// Shared-memory layout of a block: strip, tables, queue, two outboxes, the
// targets' places.
struct ClusterPlan {
  int G, H;         // blocks of the cluster, rows of a block
  int pitch;        // words of a strip row: nx + 2
  int cap;          // targets of a block in a phase at most
  int rows;         // table rows
  int dealt;        // log2 G where the rows are dealt over the blocks, else 0
  FastDiv div_pitch;  // by pitch
  unsigned off_cs, off_ap, off_queue, off_out, off_pos, bytes;
};

ClusterPlan make_plan(int nx, int ny, int ncells, int G, bool dealt) {
  ClusterPlan p;
  p.G = G;
  p.H = (ny + G - 1) / G;
  p.pitch = nx + 2;
  p.cap = (p.H / 2 + 1) * std::max(1, nx / 2);
  p.rows = ncells + 1;
  p.dealt = !dealt ? 0 : (G == 16 ? 4 : 3);
  const unsigned long long here = dealt ? (p.rows + G - 1) / G : p.rows;  // rows of a block
  p.div_pitch = fast_div_of((uint32_t)p.pitch);
  unsigned long long at = 0;
  auto take = [&](unsigned long long n) {
    const unsigned long long o = at;
    at += (n + 15) & ~15ull;
    return (unsigned)std::min<unsigned long long>(o, 0xFFFFFFF0u);
  };
  take(4ull * (p.H + 2) * p.pitch);
  p.off_cs = take(16 * here);
  p.off_ap = take(8 * here);
  p.off_queue = take(16ull * p.cap);
  p.off_out = take(2 * 16ull * p.cap);  // two 8-byte messages a copy
  p.off_pos = take(8ull * p.cap);
  p.bytes = (unsigned)std::min<unsigned long long>(at, 0xFFFFFFF0u);
  return p;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t ld_cluster(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_cluster2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ longlong2 ld_cluster2l(uint32_t addr) {
  longlong2 v;
  asm volatile("ld.shared::cluster.v2.u64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// nearest_image in 32 bits where a < 2^18 and |S| < 2^30 (coordinates and
// sides < 2^12); returns the image's number of periods + 1.
__device__ __forceinline__ uint32_t image_code(int xc, int n, int a, long long S) {
  if ((unsigned)a < (1u << 18) && S > -(1LL << 30) && S < (1LL << 30)) {
    const int d = xc * a - (int)S, half = (n * a) >> 1;  // 2 d > n a: d > n a / 2
    return d > half ? 0u : (-d > half ? 2u : 1u);
  }
  const long long img = nearest_image(xc, n, a, S);
  return img < xc ? 0u : (img > xc ? 2u : 1u);
}

// 64-bit shared-memory addition as two 32-bit ones (order-free and exact:
// every addition that wraps the low word carries one into the high word).
__device__ __forceinline__ void add64(unsigned long long* p, long long d) {
  unsigned* w = reinterpret_cast<unsigned*>(p);
  const unsigned lo = (unsigned)d;
  const unsigned old = atomicAdd(w, lo);
  const unsigned hi = (unsigned)(d >> 32) + (old + lo < old ? 1u : 0u);
  if (hi) atomicAdd(w + 1, hi);
}

// Scalars of the replica, read from shared memory in the phases: as constant
// global loads they were issued again in every phase, after a barrier that
// drops the L1 lines (600 cycles of a phase).
struct ClusterCtx {
  const float *field, *stick, *chemo;
  float T;
  unsigned fixed_mask;
  int stick_on, chemo_on, perim_on, small_targets;
};

// A slot's targets among a block's rows: target i of it lies at strip word
// ci + pos[i].x and lattice site + pos[i].y (class-2 columns: i rows down).
struct ClusterSlot {
  int n;         // targets
  uint32_t ci, site;
  int column;    // the slot's targets are one column (class 2 in x)
};

// DEALT: row r of the tables is kept by block r % G alone, at r / G, where whole
// tables do not fit (in 256^2, more than 5,700 rows).
template <bool DEALT>
__global__ void __launch_bounds__(kClusterThreads, 1)
    cluster_sweep_kernel(const __grid_constant__ SweepArgs a,
                         const __grid_constant__ ClusterPlan pl) {
  constexpr unsigned long long NSLOTS = 9;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float s_J[kMaxTypes * kJPitch];
  __shared__ TypeParams s_type[kMaxTypes];
  __shared__ ClusterCtx s_ctx;
  __shared__ ClusterSlot s_slot[9];
  __shared__ int s_off[8];  // strip offset of neighbour k
  __shared__ unsigned s_qn[2], s_out[2];  // attempts queued, messages left, by phase parity
  __shared__ uint32_t s_halo[2];  // halo rows that hold copies of the own edge rows
  __shared__ unsigned long long s_tick0;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* const strip = reinterpret_cast<uint32_t*>(smem_raw);
  longlong2* const t_cs = reinterpret_cast<longlong2*>(smem_raw + pl.off_cs);
  int2* const t_ap = reinterpret_cast<int2*>(smem_raw + pl.off_ap);
  uint4* const queue = reinterpret_cast<uint4*>(smem_raw + pl.off_queue);
  uint2* const outbox = reinterpret_cast<uint2*>(smem_raw + pl.off_out);  // [2][2 cap]
  uint2* const pos = reinterpret_cast<uint2*>(smem_raw + pl.off_pos);
  const uint32_t k0 = (uint32_t)a.seed, k1 = (uint32_t)(a.seed >> 32);
  int* err = reinterpret_cast<int*>(&a.ctl[kCtlErr]);

  const DevParams* P = a.params + __ldg(&a.reps[0].pset);
  const int nx = __ldg(&a.reps[0].nx), ny = __ldg(&a.reps[0].ny);
  const int ncells = pl.rows - 1, sp = pl.pitch;
  uint32_t* const L = a.lat + __ldg(&a.reps[0].lat_off);
  const long long cell_off = __ldg(&a.reps[0].cell_off);

  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int row0 = rank * pl.H, row1 = min(ny, row0 + pl.H);
  const int nown = max(0, row1 - row0);  // own rows (0: an idle block)

  // Load the strip, the tables and the parameters.
  if (nown > 0) {
    const int n = (nown + 2) * sp;
    for (int i = tid; i < n; i += kClusterThreads) {
      const int r = i / sp, c = i - r * sp;
      int gy = row0 - 1 + r, gx = c - 1;
      gy = gy < 0 ? ny - 1 : (gy >= ny ? 0 : gy);
      gx = gx < 0 ? nx - 1 : (gx >= nx ? 0 : gx);
      strip[i] = __ldcg(L + (long long)gy * nx + gx);
    }
  }
  // (the block's rows of the tables: local row c is row c * stride + first)
  const int stride = DEALT ? pl.G : 1, first_row = DEALT ? rank : 0;
  for (int c = tid; c * stride + first_row < pl.rows; c += kClusterThreads) {
    const long long row = cell_off + c * stride + first_row;
    const unsigned long long w = __ldcg(a.ap[0] + row);
    t_ap[c] = make_int2(unpack_area(w), unpack_perim(w));
    t_cs[c].x = __ldcg(a.cs[0] + 2 * row);
    t_cs[c].y = __ldcg(a.cs[0] + 2 * row + 1);
  }
  for (int i = tid; i < kMaxTypes * kMaxTypes; i += kClusterThreads)
    s_J[(i / kMaxTypes) * kJPitch + i % kMaxTypes] = __ldg(&P->J[i]);
  if (tid < kMaxTypes)
    s_type[tid] = {__ldg(&P->lam_area[tid]), __ldg(&P->tgt_area[tid]), __ldg(&P->lam_perim[tid]),
                   __ldg(&P->tgt_perim[tid])};
  for (int i = tid; i < pl.cap; i += kClusterThreads) {
    const int ncx = max(1, nx >> 1), j = i / ncx, c = i - j * ncx;
    pos[i] = make_uint2(2u * j * sp + 2u * c, 2u * j * nx + 2u * c);
  }
  if (tid < 9) {
    // target rows y0, y0 + 2, ... of class cy among the own ones
    const int cx = tid % 3, cy = tid / 3;
    int y0 = ny - 1, nr = cy == 2 && (ny & 1) && ny - 1 >= row0 && ny - 1 < row1;
    if (cy < 2) {
      y0 = row0 + ((row0 + cy) & 1);
      nr = max(0, (min(row1, ny - (ny & 1)) - y0 + 1) / 2);
    }
    if (nown == 0) nr = 0;
    const int x0 = cx < 2 ? cx : nx - 1;
    s_slot[tid] = {nr * class_count(nx, cx), (uint32_t)((y0 - row0 + 1) * sp + x0 + 1),
                   (uint32_t)(y0 * nx + x0), cx == 2};
  }
  if (tid < 8) s_off[tid] = ((tid + (tid >= 4)) / 3 - 1) * sp + (tid + (tid >= 4)) % 3 - 1;
  if (tid < 2) {
    if (nown > 0) {
      // the first own row is the bottom halo of the block above, the last
      // one the top halo of the block below
      const int gy = tid == 0 ? (row0 == 0 ? ny - 1 : row0 - 1) : (row1 == ny ? 0 : row1);
      const int nrank = gy / pl.H, nrows = min(ny, (nrank + 1) * pl.H) - nrank * pl.H;
      s_halo[tid] = map_rank(smem_addr(strip + (tid == 0 ? nrows + 1 : 0) * sp), nrank);
    }
  }
  if (tid < 2) s_qn[tid] = s_out[tid] = 0;
  if (tid == 0)
    s_ctx = {a.field + 2 * __ldg(&a.reps[0].lat_off), P->stick, P->chemo,
             __ldg(&P->temperature), __ldg(&P->fixed_mask), __ldg(&P->stick_on),
             __ldg(&P->chemo_on), __ldg(&P->perim_on), __ldg(&P->small_targets)};
  if (tid == 0) s_tick0 = a.tick_ptr ? __ldcg(a.tick_ptr) : a.tick0;
  // the outboxes that the warp reads (their counts, then their messages)
  uint32_t cnt_addr[kSources], out_addr[kSources];
#pragma unroll
  for (int u = 0; u < kSources; ++u) {
    const int src = min(warp * kSources + u, pl.G - 1);
    cnt_addr[u] = map_rank(smem_addr(&s_out[0]), src);
    out_addr[u] = map_rank(smem_addr(outbox), src);
  }
  cluster.sync();  // no block starts before every strip is in place

  unsigned n_eval = 0, n_acc = 0;  // of the block (thread 0), of the warp

  // Messages: one changed table row each.  x: id (24 bits), images of the
  // site on both axes (0, 1, 2: one period down, the site itself, one up;
  // 2 bits each), side (1: the cell lost the site).  y: site x (12 bits),
  // site y (12 bits), perimeter change + 8.
  auto apply = [&](const uint2& m) {
    unsigned id = m.x & 0xFFFFFFu;
    if (DEALT) {
      if ((id & (unsigned)(pl.G - 1)) != (unsigned)rank) return;
      id >>= pl.dealt;
    }
    const int sign = (m.x >> 28) & 1u ? -1 : 1;
    atomicAdd(&t_ap[id].x, sign);
    atomicAdd(&t_ap[id].y, (int)(m.y >> 24) - 8);
    const int ix = (int)(m.y & 0xFFFu) + ((int)((m.x >> 24) & 3u) - 1) * nx;
    const int iy = (int)((m.y >> 12) & 0xFFFu) + ((int)((m.x >> 26) & 3u) - 1) * ny;
    add64(reinterpret_cast<unsigned long long*>(&t_cs[id].x), sign * ix);
    add64(reinterpret_cast<unsigned long long*>(&t_cs[id].y), sign * iy);
  };
  // The messages of the phase with parity b from the warp's blocks: their
  // number, the first of each lane (loaded whether it exists or not), then
  // the rest.
  uint2 msg[kSources];
  unsigned nmsg[kSources];
  auto fetch = [&](int b) {
#pragma unroll
    for (int u = 0; u < kSources; ++u) {
      nmsg[u] = ld_cluster(cnt_addr[u] + 4u * (unsigned)b);
      msg[u] = ld_cluster2(out_addr[u] +
                           8u * (unsigned)(2 * b * pl.cap + min(lane, 2 * pl.cap - 1)));
    }
  };
  auto apply_fetched = [&](int b) {
#pragma unroll
    for (int u = 0; u < kSources; ++u) {
      const unsigned n = warp * kSources + u < pl.G ? nmsg[u] : 0u;
      if (lane < (int)n) apply(msg[u]);
      for (unsigned i = 32 + lane; i < n; i += 32)
        apply(ld_cluster2(out_addr[u] + 8u * ((unsigned)(2 * b * pl.cap) + i)));
    }
  };

  // 16 attempts, two lanes each (pair_energy).
  auto evaluate = [&](const uint4& e, bool in, uint2* out, unsigned* out_n) {
    const int side = lane & 1;
    const uint32_t s = e.z, t = e.w;
    if (max(s & 0xFFFFFFu, t & 0xFFFFFFu) > (uint32_t)ncells) {
      if (in) atomicOr(err, kErrBadId);
      in = false;
    }
    bool accepted = false;
    uint2 m = make_uint2(0, 0);
    const unsigned mask = __ballot_sync(kFull, in);
    if (in) {
      const int ci = (int)e.x;
      const uint32_t own = side ? t : s;
      const unsigned id = own & 0xFFFFFFu;
      const int type = (int)(own >> 24) & (kMaxTypes - 1);
      int2 ap;
      longlong2 cs;
      if constexpr (DEALT) {
        const int owner = (int)(id & (unsigned)(pl.G - 1));
        const unsigned at = id >> pl.dealt;
        const uint2 v = ld_cluster2(map_rank(smem_addr(t_ap + at), owner));
        ap = make_int2((int)v.x, (int)v.y);
        cs = ld_cluster2l(map_rank(smem_addr(t_cs + at), owner));
      } else {
        ap = t_ap[id];
        cs = t_cs[id];
      }
      const TypeParams tp = s_type[type];
      uint32_t nb[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) nb[k] = strip[ci + (k / 3 - 1) * sp + k % 3 - 1];
      // adhesion of the own side's configuration, in neighbour order
      float en = 0.0f;
      int cnt = 0;
      const float* J = s_J + type * kJPitch;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        if (k == 4) continue;
        const float j = J[(nb[k] >> 24) & (kMaxTypes - 1)];
        const bool same = nb[k] == own;
        en = same ? en : __fadd_rn(en, j);
        cnt += same;
      }
      if (s_ctx.stick_on && side) {
        // stickiness of the old configuration, summed in neighbour order
        // and added to its adhesion as one term
        float e_st = 0.0f;
        const float* St = s_ctx.stick + type * kMaxTypes;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          if (k == 4) continue;
          if (nb[k] != t)
            e_st = __fadd_rn(e_st, __ldg(St + ((int)(nb[k] >> 24) & (kMaxTypes - 1))));
        }
        en = __fadd_rn(en, e_st);
      }
      const int sy = (int)(__umulhi((uint32_t)ci, pl.div_pitch.mul) >> pl.div_pitch.shift);
      const int x = ci - sy * sp - 1, y = row0 + sy - 1;
      // chemotaxis, lambda of the source type, of the target type for a
      // medium source
      float chemo = 0.0f;
      if (s_ctx.chemo_on) {
        const int ts = (int)(s >> 24) & (kMaxTypes - 1), tt = (int)(t >> 24) & (kMaxTypes - 1);
        const float lam = __ldg(s_ctx.chemo + (ts ? ts : tt));
        if (lam != 0.0f)
          chemo = __fmul_rn(-lam, chemo_dot<2>(s_ctx.field, (long long)nx * ny, x, y, 0,
                                               (int)(e.y & 0xFFu), nx, ny, 1));
      }
      const int dp = side ? 2 * cnt - 8 : 8 - 2 * cnt;
      float qp, qa, ex;
      if (s_ctx.small_targets && (unsigned)(ap.x | ap.y) < kSmallTable)
        constraint_terms_small(ap.x, ap.y, dp, side ? -1 : 1, tp, qp, qa);
      else
        constraint_terms_wide(ap.x, ap.y, dp, side ? -1 : 1, tp, qp, qa);
      const float dH = pair_energy(mask, side, s != 0, t != 0, en, chemo, qp, qa, tp,
                                   s_ctx.perim_on != 0);
      if (metropolis(dH, s_ctx.T, e.y, ex)) {
        const int copy = x == 0 ? nx : (x == nx - 1 ? -nx : 0);
        if (!side) {
          // the own row, the periodic column's copy, and both in the
          // neighbour's halo if it is an edge row
          strip[ci] = s;
          if (copy) strip[ci + copy] = s;
        } else if (y == row0 || y == row1 - 1) {
          const uint32_t at = 4u * (uint32_t)(x + 1);
          if (y == row0) {
            st_cluster(s_halo[0] + at, s);
            if (copy) st_cluster(s_halo[0] + at + 4 * copy, s);
          }
          if (y == row1 - 1) {
            st_cluster(s_halo[1] + at, s);
            if (copy) st_cluster(s_halo[1] + at + 4 * copy, s);
          }
        }
        accepted = true;
        m.x = id | (image_code(x, nx, ap.x, cs.x) << 24) | (image_code(y, ny, ap.x, cs.y) << 26) |
              ((unsigned)side << 28);
        m.y = (uint32_t)x | ((uint32_t)y << 12) | ((uint32_t)(dp + 8) << 24);
      }
    }
    n_acc += __popc(__ballot_sync(kFull, accepted && side));
    const bool tell = accepted && (m.x & 0xFFFFFFu);  // (the medium has no row)
    const unsigned ball = __ballot_sync(kFull, tell);
    if (ball) {  // warp-uniform
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(out_n, (unsigned)__popc(ball));
      at = __shfl_sync(kFull, at, 0);
      // (an outbox holds two messages of every target of a phase)
      if (tell) out[at + __popc(ball & lanemask_lt())] = m;
    }
  };

  // A lane's targets base + lane, + kClusterThreads, ... of a slot: places and
  // draws (random word, its low byte the source's direction).
  constexpr int U = kRoundTargets;
  struct Draws {
    int ci[U];
    uint32_t draw[U];
  };
  auto draw_targets = [&](const ClusterSlot& sl, unsigned long long phase, int base, Draws& d) {
    uint32_t c[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = max(min(base + u * kClusterThreads + lane, sl.n - 1), 0);
      uint2 at;
      if (sl.column)  // block-uniform
        at = make_uint2(2u * i * sp, 2u * i * nx);
      else
        at = pos[i];
      d.ci[u] = (int)(sl.ci + at.x);
      c[u][0] = sl.site + at.y;
      c[u][1] = (uint32_t)phase;
      c[u][2] = a.stream0;
      c[u][3] = (uint32_t)(phase >> 32);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      philox4x32_10(c[u][0], c[u][1], c[u][2], c[u][3], k0, k1);
      d.draw[u] = (c[u][1] & 0xFFFFFF00u) | __umulhi(c[u][0], 8u);
    }
  };

  int step = 0;
  Draws first;  // of the phase at hand: drawn while the block waited for it
  ClusterSlot sl = s_slot[a.slots[0]];
  draw_targets(sl, s_tick0 * NSLOTS + (unsigned long long)a.slots[0], warp * 32, first);
  for (int mc = 0; mc < a.mcs; ++mc) {
    const unsigned long long tick = s_tick0 + (unsigned long long)mc;
    for (int si = 0; si < a.nslot_active; ++si, ++step) {
      const int cur = step & 1, prv = cur ^ 1;
      if (step > 0) fetch(prv);
      const unsigned fixed_mask = s_ctx.fixed_mask;
      // the other parity's queue was last read before the last barrier; this
      // parity's outbox was last read in the phase before
      if (tid == 0) s_qn[prv] = s_out[cur] = 0;
      // ---- queue the attempts whose source differs ------------------------
      for (int base = warp * 32; base < sl.n; base += U * kClusterThreads) {
        if (base >= U * kClusterThreads)  // (lattices of more targets per lane)
          draw_targets(sl, tick * NSLOTS + (unsigned long long)a.slots[si], base, first);
        uint32_t s[U], t[U];
        bool keep[U];
        unsigned ball[U], n = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          t[u] = strip[first.ci[u]];
          s[u] = strip[first.ci[u] + s_off[first.draw[u] & 7u]];
          keep[u] = base + u * kClusterThreads + lane < sl.n && s[u] != t[u];
          if (fixed_mask && keep[u]) {
            // a target of a fixed type never changes; a source of a fixed type
            // proposes the medium instead (src/kernels2d.cu:280-290)
            if ((fixed_mask >> ((t[u] >> 24) & (kMaxTypes - 1))) & 1u) {
              keep[u] = false;
            } else if ((fixed_mask >> ((s[u] >> 24) & (kMaxTypes - 1))) & 1u) {
              s[u] = 0u;
              keep[u] = t[u] != 0u;
            }
          }
          ball[u] = __ballot_sync(kFull, keep[u]);
          n += (unsigned)__popc(ball[u]);
        }
        if (n) {  // warp-uniform
          unsigned at = 0;
          if (lane == 0) at = atomicAdd(&s_qn[cur], n);
          at = __shfl_sync(kFull, at, 0);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (keep[u])
              queue[at + __popc(ball[u] & lanemask_lt())] =
                  make_uint4((uint32_t)first.ci[u], first.draw[u], s[u], t[u]);
            at += (unsigned)__popc(ball[u]);
          }
        }
      }
      if (step > 0) apply_fetched(prv);
      // tables as of the phase's start (DEALT: in every block), queue complete
      if (DEALT && step > 0)
        cluster.sync();
      else
        __syncthreads();
      const int nq = (int)s_qn[cur];
      for (int b = warp * 16; b < nq; b += kClusterThreads / 2) {
        const int i = b + (lane >> 1);
        evaluate(queue[i < nq ? i : b], i < nq,
                 outbox + 2 * cur * pl.cap, &s_out[cur]);
      }
      if (tid == 0) n_eval += (unsigned)nq;
      // the hardware barrier of the cluster's blocks (all co-scheduled, as the
      // threads of a block are for __syncthreads), with release and acquire
      // at cluster scope for the strips and the outboxes; the next phase's
      // first draws, which need none of them, are made in between
      cluster.barrier_arrive();
      const bool last = si + 1 == a.nslot_active;
      const int next = a.slots[last ? 0 : si + 1];
      sl = s_slot[next];
      draw_targets(sl, (tick + last) * NSLOTS + (unsigned long long)next, warp * 32, first);
      cluster.barrier_wait();
    }
    if (n_eval > (1u << 30) || n_acc > (1u << 30)) {  // (an MCS adds far less)
      if (tid == 0) atomicAdd(&a.counters[0], (unsigned long long)n_eval);
      if (lane == 0) atomicAdd(&a.counters[1], (unsigned long long)n_acc);
      n_eval = n_acc = 0;
    }
  }
  if (step > 0) {  // the last phase's messages
    fetch((step - 1) & 1);
    apply_fetched((step - 1) & 1);
  }
  if (tid == 0 && n_eval) atomicAdd(&a.counters[0], (unsigned long long)n_eval);
  if (lane == 0 && n_acc) atomicAdd(&a.counters[1], (unsigned long long)n_acc);
  if (a.tick_ptr && a.tick_advance && rank == 0 && tid == 0 && a.mcs > 0)
    *a.tick_ptr = s_tick0 + (unsigned long long)a.mcs;
  // no block leaves (or reads its tables) while messages are being read
  cluster.sync();
  for (int i = tid; i < nown * nx; i += kClusterThreads) {
    const int r = i / nx, c = i - r * nx;
    L[(long long)(row0 + r) * nx + c] = strip[(r + 1) * sp + 1 + c];
  }
  // (whole tables: each block writes its share of the rows)
  const int c0 = DEALT ? tid : rank * kClusterThreads + tid;
  for (int c = c0; c * stride + first_row < pl.rows;
       c += DEALT ? kClusterThreads : pl.G * kClusterThreads) {
    const long long row = cell_off + c * stride + first_row;
    const unsigned long long w = pack_delta(t_ap[c].x, t_ap[c].y);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      a.ap[b][row] = w;
      a.cs[b][2 * row] = t_cs[c].x;
      a.cs[b][2 * row + 1] = t_cs[c].y;
    }
  }
}

cudaLaunchConfig_t cluster_config(const ClusterPlan& p, cudaStream_t s,
                                  cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.G);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = p.bytes;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.G;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// The largest plan (8 KB are left to the static arrays).  It is also the
// function's limit, one value for every lattice: the limit belongs to the
// function on the device, and engines in other threads set it too.
constexpr int kClusterSmemMax = kSweepSmemMax - 8 * 1024;

const void* cluster_fn(bool dealt) {
  return dealt ? (const void*)cluster_sweep_kernel<true> : (const void*)cluster_sweep_kernel<false>;
}

cudaError_t cluster_attributes(const void* fn) {
  cudaError_t e =
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmemMax);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

}  // namespace

int cluster_sweep_blocks(int nx, int ny, int ncells, bool dealt) {
  if (nx < 4 || nx > 0xFFF || ny > 0xFFF) return 0;  // (12-bit coordinates in messages)
  const void* fn = cluster_fn(dealt);
  for (int G : {16, 8}) {
    const ClusterPlan p = make_plan(nx, ny, ncells, G, dealt);
    if (p.bytes > (unsigned)kClusterSmemMax) continue;
    cudaLaunchAttribute attr[1];
    int n = 0;
    if (cluster_attributes(fn) == cudaSuccess) {
      const cudaLaunchConfig_t cfg = cluster_config(p, nullptr, attr);
      if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) n = 0;
    }
    cudaGetLastError();  // (a refused size is not an error of the engine)
    if (n >= 1) return G;
  }
  return 0;
}

int cluster_sweep_threads() { return kClusterThreads; }

cudaError_t launch_cluster_sweep(const SweepArgs& a, int nx, int ny, int ncells, int G,
                                 bool dealt, cudaStream_t s) {
  const void* fn = cluster_fn(dealt);
  ClusterPlan p = make_plan(nx, ny, ncells, G, dealt);
  const cudaError_t e = cluster_attributes(fn);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<SweepArgs*>(&a), &p};
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cluster_config(p, s, attr);
  return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace gpucpm
